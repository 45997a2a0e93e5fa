"""The kernels a domain's size chooses, at the sizes where the choice turns,
against the oracle bit for bit: the update staged in shared memory from 32
zones along x3 (blocks that start inside a row and reach into five), the
Lorentz factors formed by the bound kernel up to 2e5 zones, and the fixups in
one cluster up to 2^18 zones, in their own kernels beyond."""
import numpy as np
import pytest

from harm_finalwham_b200 import torus
from harm_finalwham_b200.gpu import HarmGPU
from oracle.pyoracle import Oracle
from tests.fixtures import same
from tests.test_gpu_weno5 import problem_of

pytestmark = pytest.mark.gpu


def rough(pr, seed):
    """Noise and fast zones on the torus, so that the fixups have work."""
    rng = np.random.default_rng(seed)
    pr.p[..., 1] *= 10.0 ** rng.uniform(-1.0, 1.0, pr.p.shape[:3])
    fast = rng.random(pr.p.shape[:3]) < 0.05
    pr.p[..., 2] += fast * rng.uniform(-1.0, 1.0, pr.p.shape[:3])
    pr.p = np.ascontiguousarray(pr.p)


def boosted(pr, part):
    """A part of the zones at Lorentz factors above 3, so that the lists of
    candidates are longer than the cluster that takes them has threads."""
    fast = np.random.default_rng(9).random(pr.p.shape[:3]) < part
    g33 = pr.gcov[:pr.p.shape[0], :pr.p.shape[1], torus.CENT, 3, 3]
    pr.p[..., 4] += fast * 3.0 / np.sqrt(g33)[:, :, None]
    pr.p = np.ascontiguousarray(pr.p)


def run(n, ng=3, steps=1, part=0.0, **scheme):
    dom = torus.fm_torus(*n, ng=ng, lim=scheme.get("lim", "MC"), flux=scheme.get("flux", "HLL"), seed=21)
    pr = problem_of(dom)
    pr.timeorder = scheme.get("timeorder", 2)
    pr.utoprim = scheme.get("utoprim", "2DFINAL")
    pr.doenoflux = scheme.get("doenoflux", "NOENOFLUX")
    rough(pr, 4)
    if part:
        boosted(pr, part)
    orc = Oracle()
    orc.bound_prim(pr)
    pr.dt = 1e-5 if part else 1e-3
    q = pr.copy()
    with HarmGPU.from_problem(pr) as g:
        st = g.step_ch(steps)
        p, pf, t, dt = g.download_state()
    orc.step(q, steps)
    assert same(p, q.p), f"{int(np.count_nonzero(p != q.p))} values differ"
    assert np.array_equal(pf, q.pflag) and t == q.t and dt == q.dt
    return st


@pytest.mark.parametrize("n3", [31, 32, 33, 47])
@pytest.mark.parametrize("scheme", [{}, {"timeorder": 3, "flux": "LAXF"},
                                    {"lim": "PARA", "timeorder": 4, "utoprim": "JON", "doenoflux": "ENOFINITEVOLUME"}])
def test_update_with_long_and_short_x3(n3, scheme):
    run((9, 7, n3), steps=2, **scheme)


@pytest.mark.parametrize("n", [(63, 50, 63), (65, 49, 63), (66, 63, 63), (64, 64, 64), (65, 64, 64)])
def test_domains_around_the_size_limits(n):
    assert run(n).nfixed > 0


@pytest.mark.parametrize("part", [0.1, 0.5, 1.0])
@pytest.mark.parametrize("n", [(63, 50, 33), (200, 180, 1)])
def test_long_lists_in_one_cluster(n, part):
    st = run(n, part=part)
    assert part == 1.0 or st.nfixed > 2000


@pytest.mark.parametrize("n", [(300, 1, 1), (90, 20, 1), (40, 9, 33)])
def test_an_autotuned_choice_can_be_set_again(n):
    dom = torus.fm_torus(*n, ng=6, lim="WENO5", seed=2) if n[1] > 1 else None
    if dom is None:
        from harm_finalwham_b200 import riemann
        dom = riemann.domain(riemann.RiemannProblem(n[0], 4.0 / 3.0, np.array([1.0, 1, 0, 0, 0, 0.5, 1, 0]),
                                                    np.array([0.1, 0.1, 0, 0, 0, 0.5, -1, 0])), ng=6)
        dom.lim = "WENO5"
        dom.pflag = np.zeros(dom.p.shape[:3], dtype=np.int32)
    with HarmGPU.from_problem(problem_of(dom)) as g:
        tu = g.autotune()
        g.set_tuning({**{f: tu[f]["minb"] for f in ("flux", "weno", "update", "invert")},
                      "weno_tiles": {int(q): (v["lb"], v["lines"]) for q, v in tu["weno_tiles"].items()}})
        g.init_dt()
        g.step_ch(1)
