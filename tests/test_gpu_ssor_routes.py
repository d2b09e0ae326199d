"""FP64 SSOR sweeps (ssorflow.cu) on either side of the rules that choose
between rows over all SMs, rows in one CTA and a launch per level: bit for bit
the oracle's loop (mtj/src/no/uib/cipr/matrix/sparse/SSOR.java:143-194), and no
pattern of independent rows takes long."""
import numpy as np
import pytest
from test_gpu_block_walk import grid
from test_sweep_plan_cpu import csr

from oracle import oracle as O
from ressim_gb300 import abi, api

pytestmark = pytest.mark.gpu


def tridiagonal(n):
    i = np.arange(1, n)
    return csr(n, np.r_[i, i - 1], np.r_[i - 1, i])


def red_black(n, width):
    """Two levels: the first half couples to the second only."""
    g = np.random.Generator(np.random.PCG64(n + width))
    rows = np.repeat(np.arange(n), width)
    cols = g.integers(0, n // 2, n * width)
    return csr(n, rows, np.where(rows < n // 2, cols + n // 2, cols))


def blocks(n, size):
    """Independent dense blocks: as many levels as a block has rows."""
    rows = np.repeat(np.arange(n), size)
    cols = rows // size * size + np.tile(np.arange(size), n)
    return csr(n, rows[cols < n], cols[cols < n])


def arrow(n):
    i = np.arange(1, n)
    return csr(n, np.r_[i, 0 * i], np.r_[0 * i, i])


CHAINS = {
    "tridiagonal 25600": lambda: tridiagonal(25600),  # the most doubles one CTA holds
    "tridiagonal 25601": lambda: tridiagonal(25601),
    "four rows a level": lambda: blocks(4 * 60, 60),
    "five rows a level": lambda: blocks(5 * 60, 60),
    "2D grid": lambda: grid(40, 30, 1),
}
INDEPENDENT = {
    "diagonal": lambda: csr(4000, np.zeros(0, int), np.zeros(0, int)),
    "two levels": lambda: red_black(20000, 6),
    "two levels, 60 wide": lambda: red_black(4000, 60),
    "pairs": lambda: blocks(300, 2),
    "eight levels": lambda: blocks(4096, 8),
    "10,000 rows a level": lambda: blocks(30000, 3),
    "fewer": lambda: blocks(29990, 3),
    "arrow": lambda: arrow(3000),  # two levels, a row of 3,000 entries
}


def compare(ctx, rp, col):
    n = len(rp) - 1
    g = np.random.Generator(np.random.PCG64(11))
    rows = np.repeat(np.arange(n), np.diff(rp))
    val = g.standard_normal(len(col))
    val[rows == col] = 4.0 + np.diff(rp) * (1 + g.random(n))
    val[(rows != col) & (g.random(len(col)) < 0.05)] = -0.0
    b, x0 = g.standard_normal(n), g.standard_normal(n)
    A = api.CompRowMatrix(ctx, n, rp, col, val)
    s = api.CG(ctx, abi.PC_SSOR)
    s.set_ssor(1.3, 0.7, True)
    s.set_matrix(A)
    want = O.ssor(rp, col, val, b, x0, 1.3, 0.7, True)
    assert np.array_equal(s.apply(b, x0), want)
    ctx.set_profiling(True)
    ctx.profile_reset()
    for _ in range(5):
        assert np.array_equal(s.apply(b, x0), want)
    p = ctx.profile()
    ctx.set_profiling(False)
    s.release()
    A.release()
    return sum(v[0] for k, v in p.items() if k.startswith("ssor")) / 10


@pytest.mark.parametrize("name", list(CHAINS))
def test_chains(ctx, name):
    compare(ctx, *CHAINS[name]())


@pytest.mark.parametrize("name", list(INDEPENDENT))
def test_independent_rows(ctx, name):
    """A sweep takes 10 to 180 us here; one SM alone would take 0.1 to 4 ms, the
    arrow's row of 3,000 ordered sums apart."""
    ms = compare(ctx, *INDEPENDENT[name]())
    assert ms < (0.4 if name == "arrow" else 0.09), ms
