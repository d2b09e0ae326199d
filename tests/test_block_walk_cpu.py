"""The block walks of the ILU(0) solves (blockwalk.cu), planned on the host
and walked there against the sequential solve (MTJ's
UnitLowerCompRowMatrix.solve / UpperCompRowMatrix.solve,
mtj/src/no/uib/cipr/matrix/sparse/ILU.java:54-140): every row placed once,
every operand in its window, old enough for its phase, and not overwritten by
values staged ahead."""
import ctypes as C

import numpy as np
import pytest
from test_sweep_plan_cpu import L, csr, transpose  # noqa: F401
from test_gpu_sweeps import pattern27

from ressim_gb300 import abi


def check(L, rp, col, sweep):  # noqa: F811
    stats = np.zeros(4, np.int64)
    msg = C.create_string_buffer(256)
    st = L.rsg_block_walk_check(len(rp) - 1, abi.iptr(rp), abi.iptr(col), sweep,
                                stats.ctypes.data_as(C.POINTER(C.c_int64)), msg, 256)
    return st, stats, msg.value.decode()


@pytest.mark.parametrize("dims", [(4, 3, 2), (16, 16, 8), (48, 40, 12), (75, 61, 19), (33, 65, 3), (64, 64, 1),
                                  (7, 5, 33), (100, 3, 4), (5, 200, 2)])
@pytest.mark.parametrize("sweep", [0, 1])
def test_grid_patterns(L, dims, sweep):  # noqa: F811
    """Grids with one and several blocks of lines per plane, lines shorter
    and longer than a warp, one plane, and shapes without a line structure."""
    rp, col, _ = pattern27(*dims, seed=3)
    st, stats, msg = check(L, rp, col, sweep)
    assert st == abi.OK, msg
    ni, nj, nk = dims
    if ni >= 16 and 3 < nj <= 32:
        assert stats[0] == nk and stats[2] == ni + 2 * (nj - 1)
    elif ni >= 16 and nj > 32:
        assert nk * -(-nj // 32) <= stats[0] <= nk * (nj // 16 + 2) and stats[2] <= ni + 62


def test_irregular_patterns(L):  # noqa: F811
    """A banded random pattern with its transpose, a diagonal matrix, a
    tridiagonal one (one row per step), an arrow (one row feeds all), and a
    pattern too wide."""
    g = np.random.Generator(np.random.PCG64(8))
    n = 3000
    rows = g.integers(0, n, 6 * n)
    band = csr(n, rows, np.clip(rows + g.integers(-40, 41, len(rows)), 0, n - 1))
    far = csr(n, rows, g.integers(0, n, len(rows)))
    k = np.arange(1, n)
    for p in (band, transpose(*band), far, csr(n, k[:0], k[:0]), csr(n, k, k - 1), csr(n, k, 0 * k),
              csr(n, 0 * k, k)):
        for sweep in (0, 1):
            st, _, msg = check(L, *p, sweep)
            wide = sweep == 1 and len(p[1]) > n and p[0][1] > 60  # a row of n terms
            assert st == (abi.UNSUPPORTED if wide else abi.OK), msg
    for n in (1, 2, 33):
        rp, col = csr(n, np.arange(1, n), np.arange(n - 1))
        for sweep in (0, 1):
            assert check(L, rp, col, sweep)[0] == abi.OK
