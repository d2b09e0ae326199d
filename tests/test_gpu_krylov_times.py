"""The Krylov iteration's own kernels, against one another (so that the clock
does not matter)."""
import time

import numpy as np
import pytest
from test_gpu_sweeps import pattern27

from ressim_gb300 import abi, api

pytestmark = pytest.mark.gpu


def solver(ctx, cls, dims, its):
    """A solve of exactly `its` iterations, and the matrix's order."""
    rp, col, val = pattern27(*dims, seed=3)
    n = len(rp) - 1
    A = api.CompRowMatrix(ctx, n, rp, col, val)
    s = cls(ctx, abi.PC_DIAGONAL, rtol=1e-300, atol=1e-300, dtol=1e300, max_iter=its)
    s.set_matrix(A)
    b = np.random.Generator(np.random.PCG64(1)).standard_normal(n)
    return (lambda: s.solve(A, b, np.zeros(n), raise_on_fail=False)), (s, A)


def profiled(ctx, run):
    ctx.set_profiling(True)
    ctx.profile_reset()
    run()
    p = ctx.profile()
    ctx.set_profiling(False)
    return p


def test_chaining_does_not_cost(ctx):
    """CG on 65,536 rows, where a kernel's blocks fill the GPU once or twice:
    chained, the solve takes less than its kernels one by one (0.76 of it; 1.12
    when blocks of the next kernel started beside the running one)."""
    run, held = solver(ctx, api.CG, (64, 64, 16), 400)
    run()
    wall = []
    for _ in range(5):
        ctx.synchronize()
        t = time.perf_counter()
        run()
        wall.append(time.perf_counter() - t)
    total = sum(v[0] for v in profiled(ctx, run).values()) * 1e-3
    assert min(wall) < 0.95 * total, (min(wall), total)
    for h in held:
        h.release()


def test_reductions_keep_their_blocks_in_flight(ctx):
    """A Gram-Schmidt step reads three vectors, writes one and sums, scaling a
    vector reads one and writes one: on 524,288 rows 3.1 times as long (3.6 when
    the state of the recurrences took a third of the blocks' registers)."""
    run, held = solver(ctx, api.GMRES, (128, 128, 32), 60)
    run()
    p = profiled(ctx, run)
    per = {k: p[k][0] / p[k][1] for k in ("gm_mgs", "gm_vset")}
    assert per["gm_mgs"] < 3.35 * per["gm_vset"], per
    for h in held:
        h.release()
