"""The FP32 preconditioners inside the mixed-precision solver, entry by entry:
with an inner BiCGstab that stops at the first half of its first step, one outer
step gives x = y M^-1 b, y from a least-squares problem of one unknown, so the x
that a solve stopped there returns shows every row of one application.  The
reference is the same step in FP64 with the oracle's ILU(0)
(mtj/src/no/uib/cipr/matrix/sparse/ILU.java:54-140) or V-cycle (AMG.java).

Bounds, as a share of max |x|: a row's sum of m terms carries m + 2 roundings of
2^-24, and a triangular sweep multiplies an error by 1 / (1 - r), r the largest
share of a row's off-diagonal sum in its diagonal.  ILU(0): m up to 48, r = 1/2,
two sweeps: 50 * 2^-24 * (2 * 2 + 2) = 2e-5.  An operand taken from a wrong row
shows as its coefficient's share of the diagonal, about 1e-2 on these patterns.
V-cycle: four sweeps that damp errors on each of up to five levels, 32 roundings
a row and as many in the products between: 20 * 2 * 32 * 2^-24 = 8e-5."""
import numpy as np
import pytest
from test_gpu_block_walk import PATTERNS, grid

from oracle import oracle as O
from ressim_gb300 import abi, api

pytestmark = pytest.mark.gpu


def dominant(rp, col, seed, share):
    """Random negative couplings, the diagonal 1 / share times their sum."""
    g = np.random.Generator(np.random.PCG64(seed))
    n = len(rp) - 1
    rows = np.repeat(np.arange(n), np.diff(rp))
    val = np.where(rows == col, 0.0, -(0.5 + g.random(len(col))))
    d = np.bincount(rows, -val, n)
    val[rows == col] = np.where(d > 0, d / share, 1.0)
    return val


def one_step(rp, col, val, b, M):
    """x after one outer step from zero, in FP64."""
    A = lambda v: O.csr_op(0, rp, col, val, v)  # noqa: E731
    v = b / np.linalg.norm(b)
    ph = M(v)
    av = A(ph)
    alpha = (v @ v) / (v @ av)
    assert np.linalg.norm(v - alpha * av) < 0.8  # the inner solve stops here
    z = alpha * ph
    w = A(z)
    h = w @ v
    return np.linalg.norm(b) * h / (w @ w) * z


def returned(ctx, pc, rp, col, val, b):
    n = len(rp) - 1
    A = api.CompRowMatrix(ctx, n, rp, col, val)
    s = api.MixedFGMRES(ctx, pc, rtol=1e-300, max_iter=2, restart=1)
    s.set_inner(1, 0.9)
    s.set_matrix(A)
    xs = [s.solve(A, b, np.zeros(n), raise_on_fail=False) for _ in range(2)]
    assert s.last_info.iterations == 2 and np.array_equal(*xs)
    s.release()
    A.release()
    return xs[0]


@pytest.mark.parametrize("name", [k for k in PATTERNS if k not in ("1 row", "diagonal", "dense rows")])
def test_ilu(ctx, name):
    rp, col = PATTERNS[name]()
    val = dominant(rp, col, 3, 0.5)
    b = np.random.Generator(np.random.PCG64(4)).standard_normal(len(rp) - 1)
    want = one_step(rp, col, val, b, lambda v: O.ilu(rp, col, val, v)[1])
    assert np.max(np.abs(returned(ctx, abi.PC_ILU, rp, col, val, b) - want)) <= 2e-5 * np.max(np.abs(want))


@pytest.mark.parametrize("diagonal", [1e-42, 1e-315])
def test_ilu_scaled_rows_out_of_range(ctx, diagonal):
    """One row so small that the reciprocal of its pivot overflows, in single
    precision or in double too: the sweeps that divide last take over.  The row
    itself is left out of the comparison (its FP32 values have few bits)."""
    rp, col = grid(18, 35, 4)
    n = len(rp) - 1
    rows = np.repeat(np.arange(n), np.diff(rp))
    val = dominant(rp, col, 3, 0.5)
    b = np.random.Generator(np.random.PCG64(4)).standard_normal(n)
    lone = rows == n - 1
    val[lone & (col != n - 1)] = 0.0  # nothing else depends on the row or on what it holds
    val[(col == n - 1) & ~lone] = 0.0
    val[lone & (col == n - 1)] = diagonal
    b[n - 1] = 0.0
    s = api.BiCGstab(ctx, abi.PC_ILU, rtol=1e-12, max_iter=100)
    A = api.CompRowMatrix(ctx, n, rp, col, val)
    s.set_matrix(A)
    x = s.solve(A, b, np.zeros(n))
    _, its, _, _, _ = O.solve(abi.BICGSTAB, abi.PC_ILU, rp, col, val, b, np.zeros(n), rtol=1e-12)
    assert abs(s.last_info.iterations - its) <= 1
    assert np.linalg.norm(b - A.mult(x)) <= 1e-11 * np.linalg.norm(b)
    s.release()
    A.release()
    if np.float32(diagonal) == 0:
        return  # no FP32 factor to divide by: the mixed-precision solver has no answer, on any route
    want = one_step(rp, col, val, b, lambda v: O.ilu(rp, col, val, v)[1])
    got = returned(ctx, abi.PC_ILU, rp, col, val, b)
    assert np.max(np.abs(got - want)[:-1]) <= 2e-5 * np.max(np.abs(want))


def flow(ni, nj, nk, seed):
    """Couplings as a flow problem has them: strong across faces, weak across
    edges and corners."""
    rp, col = grid(ni, nj, nk)
    g = np.random.Generator(np.random.PCG64(seed))
    n = len(rp) - 1
    rows = np.repeat(np.arange(n), np.diff(rp))
    r, c = np.unravel_index(rows, (nk, nj, ni)), np.unravel_index(col, (nk, nj, ni))
    step = sum(np.abs(p - q) for p, q in zip(r, c))
    val = -np.choose(step, [0.0, 1.0, 0.08, 0.02]) * (0.5 + g.random(len(col)))
    val[step == 0] = 1.1 * np.bincount(rows, -val, n)
    return rp, col, val


@pytest.mark.parametrize("dims", [(24, 23, 25), (30, 30, 31), (40, 40, 33)])
def test_vcycle(ctx, dims):
    """Fine levels in slices in either precision, in FP32 only, and by rows over
    all SMs; coarse levels of wide rows in one CTA."""
    rp, col, val = flow(*dims, seed=2)
    n = len(rp) - 1
    b = 1.0 + np.random.Generator(np.random.PCG64(4)).standard_normal(n)
    amg = O.AMG(rp, col, val)
    levels = [amg.level(k) for k in range(amg.levels())]
    assert len(levels) >= 3 and max(np.diff(levels[1]["rowptr"])) > 33
    want = one_step(rp, col, val, b, lambda v: amg.apply(v, np.zeros(n)))
    assert np.max(np.abs(returned(ctx, abi.PC_AMG, rp, col, val, b) - want)) <= 8e-5 * np.max(np.abs(want))
