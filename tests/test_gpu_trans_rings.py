"""ILU.transApply (mtj/src/no/uib/cipr/matrix/sparse/ILU.java:72-78) on the
cluster walks that push their values through distributed shared memory, as
Preconditioner.apply: the sweeps over the transpose have schedules of their
own.  A process that runs no other level walk tells which walk it was.  (The
Java loop subtracts term by term from the right-hand side, the sweep their
sum: a few roundings of values below 1.)"""
import os
import subprocess
import sys

import numpy as np
import pytest
from test_gpu_sweeps import pattern27

from oracle import oracle as O
from ressim_gb300 import abi, api

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))

SCRIPT = r"""
import sys, numpy as np
sys.path.insert(0, {root!r}); sys.path.insert(0, {tests!r})
from test_gpu_sweeps import pattern27
from oracle import oracle as O
from ressim_gb300 import abi, api
ctx = api.Context(0)
for dims in ((6, 5, 4), (33, 20, 9), (64, 64, 4), (50, 40, 1)):
    rp, col, val = pattern27(*dims, seed=96)
    n = len(rp) - 1
    A = api.CompRowMatrix(ctx, n, rp, col, val)
    s = api.BiCGstab(ctx, abi.PC_ILU)
    s.set_matrix(A)
    b = np.random.Generator(np.random.PCG64(5)).standard_normal(n)
    _, xo = O.ilu(rp, col, val, b, trans=True)
    for _ in range(2):
        assert np.allclose(s.apply(b, trans=True), xo, rtol=1e-12, atol=1e-14), dims
    print("mode", api.lib().rsg_sweep_mode())
    s.release(); A.release()
ctx.close()
"""


def test_transposed_sweeps_push_their_values():
    env = {k: v for k, v in os.environ.items() if k not in ("RSG_SWEEP", "RSG_RING_CTAS")}
    r = subprocess.run([sys.executable, "-c", SCRIPT.format(root=os.path.dirname(HERE), tests=HERE)], env=env,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert r.stdout.split() == ["mode", "2"] * 4, r.stdout


def test_transpose_follows_the_pattern(ctx):
    """One solver set up for one pattern after another: transApply is that of
    the last."""
    s = api.BiCGstab(ctx, abi.PC_ILU)
    for dims in ((6, 5, 4), (20, 9, 3), (5, 4, 3)):
        rp, col, val = pattern27(*dims, seed=96)
        n = len(rp) - 1
        A = api.CompRowMatrix(ctx, n, rp, col, val)
        s.set_matrix(A)
        b = np.random.Generator(np.random.PCG64(5)).standard_normal(n)
        _, xo = O.ilu(rp, col, val, b, trans=True)
        assert np.allclose(s.apply(b, trans=True), xo, rtol=1e-12, atol=1e-14), dims
    s.release()
