"""A set-up that fails on a zero pivot leaves the solver with the factors it
had: solves and applies go on with them, as they do when the caller carries on
after the exception (ILU.java:98-125 throws)."""
import numpy as np
import pytest
from test_gpu_block_walk import band, grid, values

from ressim_gb300 import abi, api

pytestmark = pytest.mark.gpu


def singular(rp, col, val):
    """The values with a zero pivot that a later row divides by."""
    rows = np.repeat(np.arange(len(rp) - 1), np.diff(rp))
    out = val.copy()
    out[(rows == 0) & (col == 0)] = 0.0
    return out


@pytest.mark.parametrize("cls", [api.BiCGstab, api.MixedFGMRES])
@pytest.mark.parametrize("pattern", [lambda: grid(16, 36, 5), lambda: band(900, 60)], ids=["grid", "band"])
def test_earlier_factors_stay(ctx, cls, pattern):
    rp, col = pattern()
    n = len(rp) - 1
    val = values(rp, col, 3)
    b = np.random.Generator(np.random.PCG64(4)).standard_normal(n)
    A = api.CompRowMatrix(ctx, n, rp, col, val)
    for used_before in (True, False):  # with the copies of the factors made by earlier calls, and without
        s = cls(ctx, abi.PC_ILU, rtol=1e-10, max_iter=500)
        s.set_matrix(A)

        def results():
            x = s.solve(A, b, np.zeros(n))
            return x, s.last_info.iterations, s.apply(b), s.apply(b, trans=True)

        if used_before:
            want = results()
        A.set_values(singular(rp, col, val))
        with pytest.raises(api.RSGError) as e:
            s.set_matrix(A)
        assert e.value.status == abi.ZERO_PIVOT
        A.set_values(val)
        for got, ref in zip(results(), want):
            assert np.array_equal(got, ref)
        s.release()
    A.release()


def test_another_matrix_is_not_solved_with_them(ctx):
    """After a set-up for another pattern failed on a pivot the first matrix
    needs a set-up again; with it, the solver is itself."""
    rp, col = grid(16, 20, 4)
    n = len(rp) - 1
    A = api.CompRowMatrix(ctx, n, rp, col, values(rp, col, 3))
    rq, cq = grid(9, 8, 3)
    B = api.CompRowMatrix(ctx, len(rq) - 1, rq, cq, singular(rq, cq, values(rq, cq, 5)))
    b = np.random.Generator(np.random.PCG64(4)).standard_normal(n)
    s = api.BiCGstab(ctx, abi.PC_ILU, rtol=1e-10, max_iter=500)
    s.set_matrix(A)
    want = s.solve(A, b, np.zeros(n))
    with pytest.raises(api.RSGError):
        s.set_matrix(B)
    with pytest.raises(api.RSGError) as e:
        s.solve(A, b, np.zeros(n))
    assert e.value.status == abi.BAD_ARG
    s.set_matrix(A)
    assert np.array_equal(s.solve(A, b, np.zeros(n)), want)
    # a pattern that is refused before anything is prepared for it
    gap = api.CompRowMatrix(ctx, 2, np.array([0, 1, 2], np.int32), np.array([0, 0], np.int32), np.ones(2))
    with pytest.raises(api.RSGError) as e:
        s.set_matrix(gap)
    assert e.value.status == abi.MISSING_DIAGONAL
    assert np.array_equal(s.solve(A, b, np.zeros(n)), want)
    gap.release()
    for h in (s, A, B):
        h.release()
