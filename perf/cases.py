"""Measured cases of the per-zone conservative update, through the package's
public entry points.

A case is a dict of plain values; its `kind` says which call it stands for:

  step     one context advanced with the state resident on the GPU
           (HarmGPU.step_ch, or step_graph's replays of the captured step):
           Kerr tori (2D, 3D) and the 2D Bondi flow, with the reconstruction,
           Riemann flux, time order, inverter, scheme and precision named in
           the case
  host     the drop-in's use: the active zones come from host memory, one
           step, the active zones and flags go back (page-locked arrays)
  batch    uneven 1D Riemann problems of one HarmBatch advanced to their end
           time, states uploaded at the start of each pass
  utoprim  utoprim_batch: conserved to primitive variables of host arrays
           with a metric per zone
  serve    a set of 2D/3D solves submitted together to one HarmServer, which
           is polled until every result is back

Sizes are those of the benchmark and the tests, or lie between them.
"""
import ctypes
import dataclasses
import functools
import math

import numpy as np
import torch

from harm_finalwham_b200 import bondi, riemann, torus
from harm_finalwham_b200.gpu import HarmBatch, HarmGPU, HarmServer, utoprim_batch

NPR = 8
GHOSTS = {"MC": 3, "PARA": 3, "WENO5": 6}
FOREVER = 1e9  # end time of the resident solves: no pass reaches it


def _step(name, n1, n2, n3, lim="MC", flux="HLL", problem="torus", precision="fp64", timeorder=2, utoprim="2DFINAL",
          fv=False, ng=0, graph=False, steps=1, kind="step"):
    c = dict(kind=kind, problem=problem, n1=n1, n2=n2, n3=n3, lim=lim, flux=flux, precision=precision,
             timeorder=timeorder, utoprim=utoprim, fv=fv, ng=ng or GHOSTS[lim], graph=graph, steps=steps)
    return dict(name=name, **c) if name else c


def listed():
    return [
        # the reference's CPU-runnable 2D torus, one step a call with its counters: launches and latency
        _step("torus2d_64x64", 64, 64, 1),
        # a chunk of the serving loop's smallest solve: replays of the captured step
        _step("bondi2d_32x32_graph8", 32, 32, 1, problem="bondi", graph=True, steps=8),
        # odd 2D grid, the other Riemann flux, three stages
        _step("torus2d_129x67_laxf_rk3", 129, 67, 1, flux="LAXF", timeorder=3),
        # ragged 3D grid (no extent a multiple of a warp or a tile)
        _step("torus3d_97x51x33", 97, 51, 33),
        # the 3D configuration of the long parity run
        _step("torus3d_128x64x32_weno5", 128, 64, 32, lim="WENO5"),
        # the headline configuration: state larger than L2
        _step("torus3d_256x128x128_weno5", 256, 128, 128, lim="WENO5"),
        # mixed precision (FP32 reconstruction and wave speeds)
        _step("torus3d_256x128x64_mixed", 256, 128, 64, lim="WENO5", precision="mixed"),
        # the FM torus problem file's own scheme: PARA, RK4, Jon's inverter, finite volume, 11 ghosts
        _step("torus3d_128x64x32_fishmon", 128, 64, 32, lim="PARA", timeorder=4, utoprim="JON", fv=True, ng=11),
        # the drop-in: host-owned arrays in and out around each step
        _step("host_128x64x64", 128, 64, 64, kind="host"),
        # many uneven 1D Riemann problems to their end time
        dict(name="riemann1d_batch128", kind="batch", count=128, nmin=200, nmax=1000, tf=0.2, lim="MC"),
        # batched inversion of host arrays
        dict(name="utoprim_100003", kind="utoprim", zones=100003, version="2DFINAL"),
        # solves arriving together at the serving loop, to t = 2
        dict(name="serve_12", kind="serve", count=12, tf=2.0),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("step", "step", "step", "step", "step2d", "host", "batch", "utoprim", "serve"))
    if kind == "step2d":
        return _step("", _logint(rng, 24, 300), _logint(rng, 24, 200), 1, lim=rng.choice(("MC", "PARA", "WENO5")),
                     flux=rng.choice(("HLL", "LAXF")), problem=rng.choice(("torus", "bondi")),
                     timeorder=rng.choice((2, 3, 4)), utoprim=rng.choice(("2DFINAL", "JON")),
                     graph=rng.random() < 0.5, steps=rng.randint(1, 8))
    if kind in ("step", "host"):
        zones = math.exp(rng.uniform(math.log(2.0e4), math.log(1.2e6)))
        n3 = _logint(rng, 12, 96)
        n2 = max(16, int((zones / n3 / 2.0) ** 0.5 * rng.uniform(0.8, 1.2)))
        n1 = max(24, int(zones / n3 / n2))
        if kind == "host":
            return _step("", n1, n2, n3, lim=rng.choice(("MC", "WENO5")), kind="host")
        scheme = rng.choice(("plain", "plain", "mixed", "fishmon"))
        if scheme == "fishmon":
            return _step("", n1, n2, n3, lim="PARA", timeorder=4, utoprim="JON", fv=True, ng=11)
        if scheme == "mixed":
            return _step("", n1, n2, n3, lim="WENO5", precision="mixed")
        return _step("", n1, n2, n3, lim=rng.choice(("MC", "PARA", "WENO5", "WENO5")),
                     flux=rng.choice(("HLL", "HLL", "LAXF")), timeorder=rng.choice((2, 2, 3, 4)),
                     utoprim=rng.choice(("2DFINAL", "2DFINAL", "JON")), graph=rng.random() < 0.3)
    if kind == "batch":
        nmax = _logint(rng, 300, 1000)
        return dict(kind="batch", count=_logint(rng, 4, 128), nmin=200, nmax=nmax, tf=round(rng.uniform(0.05, 0.2), 3),
                    lim=rng.choice(("MC", "PARA")))
    if kind == "utoprim":
        return dict(kind="utoprim", zones=_logint(rng, 1000, 200000), version=rng.choice(("2DFINAL", "JON")))
    return dict(kind="serve", count=rng.randint(2, 12), tf=round(rng.uniform(0.5, 2.0), 2))


# --- inputs -----------------------------------------------------------------

@functools.lru_cache(maxsize=32)
def _base(problem, n1, n2, ng, a):
    """The unperturbed 2D flow; everything a seed changes is put on top."""
    if problem == "bondi":
        return bondi.bondi(n1, n2, ng=ng, noise=0.0)
    return torus.fm_torus(n1, n2, 1, ng=ng, a=a, noise=0.0)


def _domain(problem, n1, n2, n3, ng, seed, lim="MC", flux="HLL", a=0.9375):
    """A 2D or 3D solve: the axisymmetric flow with 4% noise in the internal
    energy and, in 3D, four azimuthal density modes, all from the seed."""
    base = _base(problem, n1, n2, ng, a)
    rng = np.random.default_rng([seed, n1, n2, n3])
    g3 = ng if n3 > 1 else 0
    dom = torus.Domain(n=(n1, n2, n3), ng=ng, dx=(base.dx[0], base.dx[1], 1.0 / n3), lim=lim, flux=flux, bc=base.bc,
                       gam=base.gam, cour=base.cour, tf=FOREVER)
    for f in ("gcov", "gcon", "gcovpert", "gdet", "conn", "floors"):
        setattr(dom, f, getattr(base, f))
    p = np.repeat(base.p, n3 + 2 * g3, axis=2)
    if n3 > 1:
        phi = 2 * np.pi * (np.arange(-g3, n3 + g3) + 0.5) / n3
        amp, ph = rng.random(4), rng.random(4) * 2 * np.pi
        p[..., 0] *= 1.0 + 0.02 * sum(amp[m] * np.cos((m + 1) * phi + ph[m]) for m in range(4))
    p[..., 1] *= 1.0 + 0.04 * (rng.random(p.shape[:3]) - 0.5)
    dom.p = p
    dom.pflag = np.zeros(p.shape[:3], dtype=np.int32)
    return dom


class _DeviceView:
    """A device array of the library as torch sees it; a tensor made of it
    keeps the view, and with it the context that owns the memory."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": "<f8", "version": 2}


def _prims(g):
    ptr = ctypes.c_void_p()
    rc = g.L.hgpu_device_prims(g.h, 0, ctypes.byref(ptr))
    if rc:
        raise RuntimeError(f"hgpu_device_prims: {rc}")
    t = torch.as_tensor(_DeviceView(g, ptr.value, (NPR,) + g.nt), device="cuda")
    t.context = g
    return t


def _pinned(shape, dtype):
    return torch.empty(shape, dtype=dtype, pin_memory=True).numpy()


def _utoprim_zones(n, seed):
    """Zones around a Kerr hole: metric, primitives, conserved vector (gdet
    included) and a guess near the solution, as a host loop has them."""
    rng = np.random.default_rng(seed)
    gam = 4.0 / 3.0
    x1 = np.log(1.5) + rng.random(n) * np.log(40.0 / 1.5)
    x2 = 0.02 + 0.96 * rng.random(n)
    gcov, _ = torus.gcov_mks(x1, x2, 0.9375, 0.3)
    gcon = np.linalg.inv(gcov)
    gdet = np.sqrt(np.abs(np.linalg.det(gcov)))
    pr = np.zeros((n, NPR))
    pr[:, 0] = 10.0 ** rng.uniform(-4.0, 0.0, n)
    pr[:, 1] = pr[:, 0] * 10.0 ** rng.uniform(-3.0, 0.0, n)
    d = rng.standard_normal((n, 3))
    u = d / np.sqrt(np.einsum("zi,zij,zj->z", d, gcov[:, 1:, 1:], d))[:, None]
    pr[:, 2:5] = u * rng.uniform(0.0, 3.0, n)[:, None]
    b = rng.standard_normal((n, 3))
    b /= np.sqrt(np.einsum("zi,zij,zj->z", b, gcov[:, 1:, 1:], b))[:, None]
    pr[:, 5:8] = b * np.sqrt(pr[:, 0] * 10.0 ** rng.uniform(-4.0, 0.0, n))[:, None]
    alpha = 1.0 / np.sqrt(-gcon[:, 0, 0])
    qsq = np.einsum("zi,zij,zj->z", pr[:, 2:5], gcov[:, 1:, 1:], pr[:, 2:5])
    uc = np.zeros((n, 4))
    uc[:, 0] = np.sqrt(1.0 + qsq) / alpha
    uc[:, 1:] = pr[:, 2:5] - uc[:, :1] * gcon[:, 0, 1:] * (alpha * alpha)[:, None]
    ud = np.einsum("zij,zj->zi", gcov, uc)
    bc = np.zeros((n, 4))
    bc[:, 0] = np.einsum("zi,zi->z", pr[:, 5:8], ud[:, 1:])
    bc[:, 1:] = (pr[:, 5:8] + bc[:, :1] * uc[:, 1:]) / uc[:, :1]
    bd = np.einsum("zij,zj->zi", gcov, bc)
    bsq = np.einsum("zi,zi->z", bc, bd)
    w = pr[:, 0] + gam * pr[:, 1] + bsq
    T = w[:, None] * uc[:, :1] * ud - bc[:, :1] * bd
    T[:, 0] += (gam - 1.0) * pr[:, 1] + 0.5 * bsq
    U = np.zeros((n, NPR))
    U[:, 0] = pr[:, 0] * uc[:, 0]
    U[:, 1:5] = T
    U[:, 1] += U[:, 0]
    U[:, 5:8] = pr[:, 5:8]
    U *= gdet[:, None]
    guess = pr.copy()
    guess[:, :5] *= 1.0 + 0.05 * (rng.random((n, 5)) - 0.5)
    return dict(U=U, gcov=gcov.reshape(n, 16), gcon=gcon.reshape(n, 16), gdet=gdet, guess=guess, gam=gam), pr


SERVE_GRIDS = (("torus", 64, 64, 1), ("bondi", 32, 32, 1), ("torus", 32, 32, 1), ("bondi", 64, 64, 1),
               ("torus", 64, 32, 16), ("bondi", 128, 64, 1))


def prepare(case, seed):
    if case["kind"] in ("step", "host"):
        dom = _domain(case["problem"], case["n1"], case["n2"], case["n3"], case["ng"], seed, case["lim"], case["flux"])
        dom.timeorder, dom.utoprim = case["timeorder"], case["utoprim"]
        dom.doenoflux = "ENOFINITEVOLUME" if case["fv"] else "NOENOFLUX"
        g = HarmGPU.from_problem(dom, precision=case["precision"])
        g.bound_prim()
        dt = g.init_dt()
        s = dict(case=case, g=g)
        if case["kind"] == "host":
            n = tuple(dom.n)
            s["p"] = _pinned(n + (NPR,), torch.float64)
            s["p"][...] = g.active(dom.p)
            s["out"] = _pinned(n + (NPR,), torch.float64), _pinned(n, torch.int32)
            s["dt"] = dt
        else:
            s["prims"] = _prims(g)
        return s
    if case["kind"] == "batch":
        ng = GHOSTS[case["lim"]]
        # the zone counts go with the case, the states with the seed
        ns = np.random.default_rng(case["count"]).integers(case["nmin"], case["nmax"] + 1, case["count"])
        probs = [dataclasses.replace(q, n=int(n)) for q, n in zip(riemann.draw(case["count"], seed=seed), ns)]
        b = HarmBatch([q.n for q in probs], [q.dx for q in probs], [q.gam for q in probs], [case["tf"]] * len(probs),
                      ng=ng, lim=case["lim"], flux="HLL", cour=0.5)
        b.upload_geometry(*riemann.minkowski_geometry(b.nt[0]))
        line = b.join([riemann.primitives(q, ng) for q in probs])
        b.upload_state(line, None, 0.0, 0.0)
        b.init_dt()
        return dict(case=case, g=b, line=line, t=np.zeros(len(probs)), dt=b.status()[1].copy(), prims=_prims(b))
    if case["kind"] == "utoprim":
        return dict(case=case, **_utoprim_zones(case["zones"], seed)[0])
    doms = []
    for q in range(case["count"]):
        problem, n1, n2, n3 = SERVE_GRIDS[q % len(SERVE_GRIDS)]
        doms.append(_domain(problem, n1, n2, n3, 3, seed * 64 + q))
    return dict(case=case, server=HarmServer(int(32e9), max_active=32, steps_per_chunk=8), doms=doms)


def run(s):
    case = s["case"]
    if case["kind"] == "step":
        g = s["g"]
        st = (g.step_graph if case["graph"] else g.step_ch)(case["steps"])
        if case["precision"] != "fp64":
            return [s["prims"]]
        return [s["prims"], st.newton_iters, st.nfail, st.nfixed]
    if case["kind"] == "host":
        g = s["g"]
        g.upload_active(s["p"], 0.0, s["dt"])
        g.step_ch(1)
        p, flags, t, dt = g.download_active(s["out"])
        return [p, flags, t, dt]
    if case["kind"] == "batch":
        b = s["g"]
        b.upload_state(s["line"], None, 0.0, 0.0)
        b.set_time(s["t"], s["dt"])
        _steps, _ms, per, _fin = b.run(25)
        return [s["prims"], per]
    if case["kind"] == "utoprim":
        pr, pflag, iters = utoprim_batch(s["U"], s["gcov"], s["gcon"], s["gdet"], s["guess"], s["gam"], 2500.0,
                                         version=case["version"])
        return [pr, pflag, iters]
    srv = s["server"]
    ids = [srv.submit(d, case["tf"]) for d in s["doms"]]
    pending = len(ids)
    while pending:
        waiting, active, finished = srv.poll()
        pending = waiting + active
    out = []
    for rid in ids:
        p, flags, t, steps, _queue_ms, _run_ms = srv.result(rid)
        out.append([p, flags, t, steps])
        srv.release(rid)
    return out


# --- what a pass cannot do without -------------------------------------------

# FP64 operations (a division or a root is one) of the scheme per zone and
# stage: reconstruction and two Riemann states per face and direction, the
# conserved update with the source term, the inversion (about five Newton
# steps)
_RECON = {"MC": 150, "PARA": 450, "WENO5": 1700}
_FACE, _UPDATE, _INVERT = 900, 900, 500


def _flops(lim, ndim, stages):
    return stages * (ndim * (_RECON[lim] + _FACE) + _UPDATE + _INVERT)


def work(case):
    if case["kind"] in ("step", "host"):
        zones = case["n1"] * case["n2"] * case["n3"]
        ndim = sum(case[k] > 1 for k in ("n1", "n2", "n3"))
        # per stage: read p_b and p^n, write p_f and the flag (the finite-volume scheme: the conserved state too)
        per = case["timeorder"] * (3 * 64 + 4 + (64 if case["fv"] else 0))
        w = {"bytes": zones * per * case["steps"],
             "flops": zones * _flops(case["lim"], ndim, case["timeorder"]) * case["steps"]}
        if case["kind"] == "host":
            w["bytes"] += zones * (64 + 64 + 4)
        return w
    if case["kind"] == "batch":
        # CFL 0.5 with wave speeds near that of light: about 2 tf N steps of an N-zone problem
        n = 0.5 * (case["nmin"] + case["nmax"])
        updates = case["count"] * n * 2.0 * case["tf"] * n
        return {"bytes": updates * 2 * 196, "flops": updates * _flops(case["lim"], 1, 2)}
    if case["kind"] == "utoprim":
        return {"bytes": case["zones"] * (8 * (8 + 32 + 1 + 8 + 8) + 4), "flops": case["zones"] * _INVERT}
    total = {"bytes": 0.0, "flops": 0.0}
    for q in range(case["count"]):
        _problem, n1, n2, n3 = SERVE_GRIDS[q % len(SERVE_GRIDS)]
        # dt is about half a zone of the inner radial grid
        updates = n1 * n2 * n3 * case["tf"] * 0.7 * n1
        total["bytes"] += updates * 2 * 196
        total["flops"] += updates * _flops("MC", 3 if n3 > 1 else 2, 2)
    return total


def exact(case, seed):
    """The inversion's solution is the state its conserved vector was formed
    from; a step of the nonlinear scheme has no such closed form."""
    if case["kind"] != "utoprim":
        return None
    return [_utoprim_zones(case["zones"], seed)[1], None, None]
