"""The block walks inside the Krylov solvers (blockwalk.cu): BiCGstab and the
mixed-precision solver with ILU(0) on patterns at the edges of the walks'
range.  A wrong operand would make another preconditioner, so besides the
residual the iteration count is held to the oracle's (MTJ's BiCGstab + ILU,
mtj/src/no/uib/cipr/matrix/sparse/BiCGstab.java:65-116, ILU.java:54-140).

Bounds: a solve stops at a relative residual of 1e-12 by its recurrence, and
the true residual of these diagonally dominant systems (condition below 1e3)
strays from that by rounding only, some 1e-14: 1e-11 leaves a factor of ten.
Iterations may differ by one for the rounding of another summation order."""
import numpy as np
import pytest
from test_gpu_sweeps import pattern27
from test_sweep_plan_cpu import csr

from oracle import oracle as O
from ressim_gb300 import abi, api

pytestmark = pytest.mark.gpu


def values(rp, col, seed):
    g = np.random.Generator(np.random.PCG64(seed))
    rows = np.repeat(np.arange(len(rp) - 1), np.diff(rp))
    val = -g.random(len(col))
    d = np.zeros(len(rp) - 1)
    np.add.at(d, rows, -val)
    val[rows == col] = d + 0.3
    return val


def grid(*dims):
    rp, col, _ = pattern27(*dims, seed=3)
    return rp, col


def band(n, half):
    """Random columns within the band; every row reaches the last column (the
    elimination never looks past a row's end, which the library refuses)."""
    g = np.random.Generator(np.random.PCG64(8))
    rows = g.integers(0, n, 6 * n)
    cols = np.clip(rows + g.integers(-half, half + 1, len(rows)), 0, n - 1)
    return csr(n, np.r_[rows, 0:n], np.r_[cols, np.full(n, n - 1)])


PATTERNS = {
    "1 row": lambda: csr(1, np.zeros(0, int), np.zeros(0, int)),
    "diagonal": lambda: csr(700, np.zeros(0, int), np.zeros(0, int)),
    "tridiagonal": lambda: csr(1500, np.r_[1:1500, 0:1499], np.r_[0:1499, 1:1500]),
    "one block": lambda: grid(16, 16, 1),
    "plane per block": lambda: grid(17, 32, 5),
    "33 lines": lambda: grid(20, 33, 4),
    "blocks cut across planes": lambda: grid(33, 70, 7),
    "short lines": lambda: grid(5, 200, 2),
    "no line structure": lambda: grid(3, 3, 60),
    "2D": lambda: grid(70, 65, 1),
    "band": lambda: band(3000, 40),
    "wide band": lambda: band(2000, 300),
    "far columns": lambda: band(2500, 2500),
    "dense rows": lambda: csr(120, *[a.ravel() for a in np.indices((120, 120))]),
}


@pytest.mark.parametrize("name", list(PATTERNS))
def test_patterns(ctx, name):
    rp, col = PATTERNS[name]()
    n = len(rp) - 1
    val = values(rp, col, n)
    b = np.random.Generator(np.random.PCG64(n)).standard_normal(n)
    A = api.CompRowMatrix(ctx, n, rp, col, val)
    for cls in (api.BiCGstab, api.MixedFGMRES):
        s = cls(ctx, abi.PC_ILU, rtol=1e-12, max_iter=500)
        for _ in range(2):  # again from the state the first solve left
            s.set_matrix(A)
            x = s.solve(A, b, np.zeros(n))
            assert np.linalg.norm(b - A.mult(x)) <= 1e-11 * np.linalg.norm(b)
        if cls is api.BiCGstab:
            _, its, _, _, _ = O.solve(abi.BICGSTAB, abi.PC_ILU, rp, col, val, b, np.zeros(n), rtol=1e-12)
            assert abs(s.last_info.iterations - its) <= 1
        s.release()
    A.release()


def test_not_a_number_does_not_stall(ctx):
    """A right-hand side with a NaN, also one with the very bits that mark an
    unwritten value between blocks: the solve ends as MTJ's does on NaN (it
    never converges), not in a wait."""
    rp, col = grid(20, 40, 4)
    n = len(rp) - 1
    A = api.CompRowMatrix(ctx, n, rp, col, values(rp, col, 1))
    for bits in (0x7FF8000000000000, 0xFFF4DEAD5EED0BAD):
        b = np.ones(n)
        b[37] = np.array([bits], np.uint64).view(np.float64)[0]
        s = api.BiCGstab(ctx, abi.PC_ILU, rtol=1e-10, max_iter=20)
        s.set_matrix(A)
        with pytest.raises(api.RSGError) as e:
            s.solve(A, b, np.zeros(n))
        assert e.value.status in (1, 2, 3)
        s.release()
    # and the next solve on the same solver is not affected
    s = api.BiCGstab(ctx, abi.PC_ILU, rtol=1e-10, max_iter=200)
    s.set_matrix(A)
    b[37] = np.nan
    s.solve(A, b, np.zeros(n), raise_on_fail=False)
    b[37] = 1.0
    x = s.solve(A, b, np.zeros(n))
    assert np.linalg.norm(b - A.mult(x)) <= 1e-9 * np.linalg.norm(b)
    s.release()
    A.release()
