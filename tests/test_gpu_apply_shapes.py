"""Preconditioner.apply of ILU(0) settles on the faster cluster shape of its
level walks, sweep by sweep, where its first calls can tell them apart."""
import numpy as np
import pytest
from test_gpu_sweeps import pattern27

from ressim_gb300 import abi, api

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(64, 64, 8), (96, 96, 12), (128, 128, 8), (6, 5, 4)])
def test_faster_shape_is_taken(ctx, dims):
    """A shape counts as the faster when its mean over ten calls is 3% below
    the other's (repeated means differ by 0.5%)."""
    rp, col, val = pattern27(*dims, seed=3)
    n = len(rp) - 1
    b = np.random.Generator(np.random.PCG64(5)).standard_normal(n)
    A = api.CompRowMatrix(ctx, n, rp, col, val)
    ms, out = {}, []
    for shape in (16, 8):
        s = api.BiCGstab(ctx, abi.PC_ILU)
        s.set_walk_shape(shape)
        s.set_matrix(A)
        out.append(s.apply(b))
        ctx.set_profiling(True)
        ctx.profile_reset()
        for _ in range(10):
            s.apply(b)
        p = ctx.profile()
        ctx.set_profiling(False)
        assert s.walk_shapes()[:2] == [shape, shape]
        ms[shape] = [p[k][0] / p[k][1] for k in ("ilu_lower", "ilu_upper")]
        s.release()
    s = api.BiCGstab(ctx, abi.PC_ILU)
    for _ in range(2):  # new values keep the choice
        s.set_matrix(A)
        for _ in range(7):
            out.append(s.apply(b))
        for k, got in enumerate(s.walk_shapes()[:2]):
            fast, slow = sorted((8, 16), key=lambda c: ms[c][k])
            if ms[fast][k] < 0.97 * ms[slow][k]:
                assert got == fast, (k, ms)
    s.release()
    A.release()
    assert all(np.array_equal(x, out[0]) for x in out)
