"""fluxcalc on the GPU against the oracle on drawn states: every face flux
the update reads, and the three dt estimates, bit for bit (up to the sign of
zero).  The states reach what the torus's flow rarely does: jumps in every
primitive, constant stretches, exact zeros, and fields from 1e-30 down into
the denormals, where shared reciprocals and the indicators read from
exponents give way to the plain expressions, and infinities, whose products
with zeros the kernels leave out.  WENO5 runs with segments of
many lengths: one cell, remainders, a whole line."""
import numpy as np
import pytest

from harm_finalwham_b200 import torus
from harm_finalwham_b200.gpu import HarmGPU, HarmGPUError
from oracle.pyoracle import Oracle
from tests.fixtures import same
from tests.test_gpu_weno5 import problem_of
from tests.test_oracle_flux_reference import draw_flux_state

pytestmark = pytest.mark.gpu


def draw(pr, kind, seed):
    draw_flux_state(pr, 900 + seed)
    rng = np.random.default_rng(seed)
    if kind == "zeros":
        for v in (2, 3, 4, 5, 6, 7):
            pr.p[..., v] *= rng.random(pr.p.shape[:3]) < 0.5
        pr.p[:, : pr.p.shape[1] // 3, :, 5:] = 0.0
        pr.p[..., 3] *= -1.0
    if kind == "tiny":
        # each field at its own scale, from normal to denormal
        for v in (5, 6, 7):
            pr.p[..., v] *= 10.0 ** rng.choice([0, -30, -100, -160, -250, -305, -318], size=pr.p.shape[:3])
    if kind == "constant":
        pr.p[...] = pr.p[:1, :1, :1]
        pr.p[pr.p.shape[0] // 2:, ..., 0] *= 1.0 + 1e-13
        pr.p[:, pr.p.shape[1] // 2:, :, 1] *= 1.0 + 3e-13
    pr.p = np.ascontiguousarray(pr.p)


def check(pr, tiles=None):
    err, F, ndt = Oracle().fluxcalc(pr)
    assert err == 0
    with HarmGPU.from_problem(pr) as g:
        if tiles:
            g.set_tuning({"flux": 4, "weno": 3, "update": 3, "invert": 1,
                          "weno_tiles": {d + 1: (min(tiles, pr.n[d] + 2), 8) for d in range(3) if pr.n[d] > 1}})
        G, gdt = g.fluxcalc()
    for d in range(3):
        if pr.n[d] == 1:
            continue
        sl = tuple(slice(q, q + n + (1 if a == d else 0)) for a, (q, n) in enumerate(zip(pr.g, pr.n)))
        a, b = G[d][sl], F[d][sl]
        assert same(a, b), f"dir {d + 1}: {int(np.count_nonzero(a != b))} of {a.size} fluxes differ"
    assert [gdt[d] for d in range(3) if pr.n[d] > 1] == [ndt[d] for d in range(3) if pr.n[d] > 1]


@pytest.mark.parametrize("kind", ["jumps", "zeros", "tiny", "constant"])
@pytest.mark.parametrize("lim,flux", [("WENO5", "HLL"), ("MC", "HLL"), ("PARA", "LAXF")])
@pytest.mark.parametrize("n", [(19, 13, 11), (24, 17, 1)])
def test_fluxes_of_drawn_states_match_oracle(n, lim, flux, kind):
    dom = torus.fm_torus(*n, ng=6, lim=lim, flux=flux, seed=3)
    pr = problem_of(dom)
    draw(pr, kind, 1)
    check(pr)


# values whose fluxes are not finite though every wave speed is
ODD = [(n, v, value) for n in [(19, 13, 11), (24, 17, 1)]
       for v, value in [(0, np.inf), (1, 1e308), (1, -1e308), (6, np.inf), (7, np.nan)]]
ODD += [((24, 17, 1), 1, -np.inf), ((24, 17, 1), 5, 1e308)]


@pytest.mark.parametrize("lim,flux", [("WENO5", "HLL"), ("MC", "HLL"), ("PARA", "LAXF")])
@pytest.mark.parametrize("n,v,value", ODD)
def test_fluxes_that_are_not_finite_match_oracle(n, v, value, lim, flux):
    dom = torus.fm_torus(*n, ng=6, lim=lim, flux=flux, seed=3)
    pr = problem_of(dom)
    draw(pr, "jumps", 1)
    pr.p[np.random.default_rng(1).random(pr.p.shape[:3]) < 0.01, v] = value
    check(pr)


@pytest.mark.parametrize("scheme", [{}, {"timeorder": 3}, {"timeorder": 4}, {"timeorder": 4, "doenoflux": "ENOFINITEVOLUME"}])
@pytest.mark.parametrize("v,value", [(0, 1.7e308), (1, 1e308), (5, np.nan), (7, np.inf)])
@pytest.mark.parametrize("n", [(24, 17, 1), (12, 9, 33)])
def test_a_zone_that_failed_in_one_stage_fails_as_the_oracles(n, v, value, scheme):
    """0 times an infinity or NaN of an earlier stage is NaN: the scheme's
    zero weights keep the zone failing in the later ones."""
    dom = torus.fm_torus(*n, ng=6, lim="MC", flux="HLL", seed=3)
    pr = problem_of(dom)
    pr.timeorder = scheme.get("timeorder", 2)
    pr.doenoflux = scheme.get("doenoflux", "NOENOFLUX")
    pr.p[pr.g[0] + 8, pr.g[1] + 6, pr.g[2] + n[2] // 2, v] = value
    pr.p = np.ascontiguousarray(pr.p)
    orc = Oracle()
    orc.bound_prim(pr)
    pr.dt = 1e-3
    q = pr.copy()
    with HarmGPU.from_problem(pr) as g:
        if scheme.get("doenoflux"):
            # the conserved state of the zone itself
            q.u = orc.pi2u(q)
        st = orc.step(q, 1)
        if st.err:
            with pytest.raises(HarmGPUError):
                g.step_ch(1)
            return
        g.step_ch(1)
        p, pf, _t, _dt = g.download_state()
    assert np.count_nonzero(q.pflag) > 0
    assert same(p, q.p) and np.array_equal(pf, q.pflag)


@pytest.mark.parametrize("lb", [1, 2, 7, 8, 9, 64])
@pytest.mark.parametrize("n", [(19, 13, 11), (24, 17, 1)])
def test_weno5_segments_of_any_length(n, lb):
    dom = torus.fm_torus(*n, ng=6, lim="WENO5", flux="HLL", seed=5)
    pr = problem_of(dom)
    draw(pr, "jumps", 2)
    check(pr, tiles=lb)
