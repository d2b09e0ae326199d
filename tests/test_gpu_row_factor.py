"""ILU(0) factorisation by rows (factor.cu) against the oracle's sequential
loop (mtj/src/no/uib/cipr/matrix/sparse/ILU.java:98-125), bit for bit through
Preconditioner.apply: rows up to a warp's 32 entries, longer ones (factorised
by levels instead), and values over the exponent range in which the quotients
are corrected from reciprocals and beyond it."""
import numpy as np
import pytest
from test_gpu_block_walk import PATTERNS, grid, values
from test_sweep_plan_cpu import csr

from oracle import oracle as O
from ressim_gb300 import abi, api

pytestmark = pytest.mark.gpu


def check(ctx, rp, col, val):
    n = len(rp) - 1
    A = api.CompRowMatrix(ctx, n, rp, col, val)
    s = api.BiCGstab(ctx, abi.PC_ILU)
    b = np.random.Generator(np.random.PCG64(5)).standard_normal(n)
    _, xo = O.ilu(rp, col, val, b)
    for _ in range(2):
        s.set_matrix(A)
        assert np.array_equal(s.apply(b), xo, equal_nan=True)
    s.release()
    A.release()


@pytest.mark.parametrize("name", list(PATTERNS))
def test_patterns(ctx, name):
    rp, col = PATTERNS[name]()
    check(ctx, rp, col, values(rp, col, 7))


@pytest.mark.parametrize("decades", [3, 60, 150])
def test_value_range(ctx, decades):
    """Rows scaled over +-decades (the quotients then span twice that: the
    last range takes plain divisions too), zeros and negative zeros among the
    entries off the diagonal."""
    rp, col = grid(9, 8, 5)
    rows = np.repeat(np.arange(len(rp) - 1), np.diff(rp))
    g = np.random.Generator(np.random.PCG64(decades))
    val = values(rp, col, decades)
    off = rows != col
    val[off & (g.random(len(col)) < 0.1)] = 0.0
    val[off & (g.random(len(col)) < 0.05)] = -0.0
    check(ctx, rp, col, val * (10.0 ** g.uniform(-decades, decades, len(rp) - 1))[rows])


def test_row_lengths_around_a_warp(ctx):
    """The longest row has 30, 32 and 34 entries."""
    for width in (15, 16, 17):
        n = 400
        i = np.arange(n)
        rows = np.concatenate([i] * (2 * width - 1))
        cols = np.concatenate([np.clip(i + d, 0, n - 1) for d in range(1 - width, width)])
        rp, col = csr(n, np.r_[rows, i], np.r_[cols, np.full(n, n - 1)])
        check(ctx, rp, col, values(rp, col, width))
