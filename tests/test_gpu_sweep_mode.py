"""rsg_sweep_mode names the walks that have run: a process whose solves ran
block walks is not undecided."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))

SCRIPT = r"""
import sys, numpy as np
sys.path.insert(0, {root!r}); sys.path.insert(0, {tests!r})
from test_gpu_sweeps import pattern27
from ressim_gb300 import abi, api
modes = [api.lib().rsg_sweep_mode()]
ctx = api.Context(0)
rp, col, val = pattern27(9, 8, 4, seed=1)
n = len(rp) - 1
A = api.CompRowMatrix(ctx, n, rp, col, val)
s = api.BiCGstab(ctx, abi.PC_ILU)
s.set_matrix(A)
s.solve(A, np.ones(n), np.zeros(n))
modes.append(api.lib().rsg_sweep_mode())
s.apply(np.ones(n))
modes.append(api.lib().rsg_sweep_mode())
print(*modes)
s.release(); A.release(); ctx.close()
"""


@pytest.mark.parametrize("sweep,modes", [(None, "-1 3 2"), ("ring", "-1 2 2"), ("pipelined", "-1 1 1")])
def test_modes(sweep, modes):
    env = {k: v for k, v in os.environ.items() if k not in ("RSG_SWEEP", "RSG_RING_CTAS")}
    if sweep:
        env["RSG_SWEEP"] = sweep
    r = subprocess.run([sys.executable, "-c", SCRIPT.format(root=os.path.dirname(HERE), tests=HERE)], env=env,
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == modes, r.stdout + r.stderr
