"""bench.py's byte counts of the conserved update follow the library's own
Runge-Kutta tables: which accumulators a stage reads."""
import os
import re

import pytest

import bench

SRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "harm_finalwham_b200", "csrc", "harm_gpu.cu")


def stages(order):
    table = re.search(rf"kRK{order}\[{order}\] = (.*?);", open(SRC).read(), re.S).group(1)
    num = [eval(v, {}) for v in re.findall(r"\d+\.\d+(?: / \d+\.\d+)?", table)]  # noqa: S307
    assert len(num) == 6 * order
    return [(num[6 * s:6 * s + 3], num[6 * s + 3:6 * s + 6]) for s in range(order)]


@pytest.mark.parametrize("order", [1, 2, 3, 4])
def test_reads_follow_the_tables(order):
    reads, left = [], False
    for s, (cuf, cun) in enumerate(stages(order)):
        reads.append((int(s > 0 and cuf[1] != 0), int(left)))
        left = left or any(cun)
    assert bench.RK_READS[order] == reads


def test_midpoint_update_moves_336_bytes_a_zone():
    # p_b 64, fluxes 120, EMFs 24, uf and ucum 128; then p^n instead of uf
    assert bench.update_bytes(3, 2, False) == 336
