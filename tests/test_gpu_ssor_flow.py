"""SSOR sweeps as a dataflow of rows (ssorflow.cu) against the oracle's
sequential loop (mtj/src/no/uib/cipr/matrix/sparse/SSOR.java:143-194), bit for
bit through Preconditioner.apply: a thread per row up to 32 entries beside the
diagonal while the vector fits shared memory, else a warp per row (up to 128
entries in registers, longer rows beyond), in one CTA up to 4096 rows and over
all SMs above."""
import numpy as np
import pytest
from test_gpu_block_walk import grid

from oracle import oracle as O
from ressim_gb300 import abi, api

pytestmark = pytest.mark.gpu


def scattered(n, width, seed, near=400):
    """Rows of `width` entries beside the diagonal (fewer at the ends), within `near` columns."""
    g = np.random.Generator(np.random.PCG64(seed))
    rp, col = [0], []
    for i in range(n):
        around = np.setdiff1d(np.arange(max(0, i - near), min(n, i + near + 1)), [i])
        c = g.choice(around, min(width, len(around)), replace=False)
        col.append(np.sort(np.append(c, i)))
        rp.append(rp[-1] + len(col[-1]))
    return np.array(rp, np.int32), np.concatenate(col).astype(np.int32)


PATTERNS = {
    "one row": lambda: scattered(1, 0, 1),
    "31 rows": lambda: scattered(31, 5, 2),
    "33 rows of 32": lambda: scattered(33, 32, 3),
    "1000 rows of 32": lambda: scattered(1000, 32, 4),
    "200 rows of 33": lambda: scattered(200, 33, 5),
    "700 rows of 128": lambda: scattered(700, 128, 6),
    "500 rows of 250": lambda: scattered(500, 250, 7),
    "4096 rows of 40": lambda: scattered(4096, 40, 8, near=100),
    "4097 rows of 40": lambda: scattered(4097, 40, 9, near=100),
    "lower only": lambda: _triangle(300, 20, True),
    "upper only": lambda: _triangle(300, 40, False),
    "grid 24x23x25": lambda: grid(24, 23, 25),
    "grid 30x30x31": lambda: grid(30, 30, 31),  # more doubles than shared memory takes
}


def _triangle(n, width, lower):
    rp, col = scattered(n, width, 10)
    keep = [c[(c <= i) if lower else (c >= i)] for i in range(n) for c in [col[rp[i]:rp[i + 1]]]]
    return np.concatenate([[0], np.cumsum([len(c) for c in keep])]).astype(np.int32), np.concatenate(keep).astype(np.int32)


@pytest.mark.parametrize("name", list(PATTERNS))
@pytest.mark.parametrize("reverse", [True, False])
def test_matches_sequential_loop(ctx, name, reverse):
    rp, col = PATTERNS[name]()
    n = len(rp) - 1
    g = np.random.Generator(np.random.PCG64(11))
    val = g.standard_normal(len(col))
    rows = np.repeat(np.arange(n), np.diff(rp))
    val[col == rows] = 4.0 + np.diff(rp) * (1 + g.random(n))
    val[g.random(len(col)) < 0.02] *= -0.0
    val[col == rows] = np.where(val[col == rows] == 0, 5.0, val[col == rows])
    b, x0 = g.standard_normal(n), g.standard_normal(n)
    A = api.CompRowMatrix(ctx, n, rp, col, val)
    s = api.CG(ctx, abi.PC_SSOR)
    s.set_ssor(1.3, 0.7, reverse)
    s.set_matrix(A)
    want = O.ssor(rp, col, val, b, x0, 1.3, 0.7, reverse)
    for _ in range(2):
        assert np.array_equal(s.apply(b, x0), want)
    s.release()
    A.release()
