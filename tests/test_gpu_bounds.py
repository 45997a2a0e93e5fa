"""Boundaries whose x2 sides differ, one of them a pole: the other side's
ghosts take the pole's row as it was before the pole zeroes u~2 and B2 there
(the order of the reference's fills: ghosts first, then the row)."""
import numpy as np
import pytest

from harm_finalwham_b200 import torus
from harm_finalwham_b200.gpu import HarmGPU
from tests.test_gpu_weno5 import problem_of

pytestmark = pytest.mark.gpu

PERIODIC, POLE, FLIP = 7, 4, 1001


@pytest.mark.parametrize("up,dn", [(PERIODIC, POLE), (POLE, PERIODIC), (FLIP, POLE), (POLE, FLIP)])
@pytest.mark.parametrize("n", [(96, 3, 64), (40, 3, 1), (64, 48, 32)])
def test_a_pole_beside_another_boundary(n, up, dn):
    ng = 3
    dom = torus.fm_torus(*n, ng=ng, lim="MC", flux="HLL", seed=3)
    rng = np.random.default_rng(4)
    dom.p[..., 2:] += 1e-3 * rng.standard_normal(dom.p[..., 2:].shape)
    pr = problem_of(dom)
    bc = list(pr.bc)
    bc[2], bc[3] = up, dn
    pr.bc = tuple(bc)
    act = (slice(ng, -ng), slice(ng, -ng), slice(ng, -ng) if n[2] > 1 else slice(None))
    with HarmGPU.from_problem(pr) as g:
        g.bound_prim()
        p = g.download_state()[0]
    before = pr.p[act]
    inner = p[act[0], :, act[2]]

    def source(j):
        """The row of a ghost or active row j, and what its side does to u~2 and B2."""
        if j < 0:
            side, row = dn, (j + n[1] if dn == PERIODIC else -j - 1)
        elif j >= n[1]:
            side, row = up, (j - n[1] if up == PERIODIC else 2 * n[1] - 1 - j)
        else:
            side, row = None, j
        return row, {FLIP: -1.0, POLE: 0.0}.get(side, 1.0)

    for j in range(-ng, n[1] + ng):
        row, factor = source(j)
        if (dn == POLE and j <= 0) or (up == POLE and j >= n[1] - 1):
            factor = 0.0
        want = before[:, row].copy()
        want[..., [3, 6]] *= factor
        assert np.array_equal(inner[:, ng + j], want), f"row {j}"
