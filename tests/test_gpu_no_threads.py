"""Where the process can have no further host threads, the ILU(0) analysis of a
large pattern plans in the calling thread and an ensemble is stepped by it."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))

SCRIPT = r"""
import sys, ctypes, numpy as np
sys.path.insert(0, {root!r}); sys.path.insert(0, {tests!r})
from test_gpu_block_walk import grid, values
from ressim_gb300 import abi, api, workloads as W
threads = ctypes.CDLL({shim!r})
ctx = api.Context(0)
rp, col = grid(40, 40, 10)
n = len(rp) - 1
assert len(col) > 200000
A = api.CompRowMatrix(ctx, n, rp, col, values(rp, col, 1))
b = np.ones(n)
xs, states = [], []
for deny in (0, 1):
    s = api.BiCGstab(ctx, abi.PC_ILU, rtol=1e-10, max_iter=500)
    threads.deny_threads(deny)
    s.set_matrix(A)
    threads.deny_threads(0)
    xs.append(s.solve(A, b, np.zeros(n)))
    s.release()
    ctxs = [api.Context(0) for _ in range(3)]
    sims = [W.build_two_phase_sim(c, 12 + k, 10, 4, seed=k, rtol=1e-10)[0] for k, c in enumerate(ctxs)]
    threads.deny_threads(deny)
    _, sts = api.ensemble_step_batched(sims, [8640.0] * 3)
    threads.deny_threads(0)
    assert not sts.any(), sts
    states.append([s.state()[0].copy() for s in sims])
    for c in ctxs:
        c.close()
assert np.array_equal(*xs)
assert all(np.array_equal(p, q) for p, q in zip(*states))
print("denied", threads.threads_denied())
"""


def test_no_further_threads(tmp_path):
    shim = str(tmp_path / "deny_threads.so")
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", shim, os.path.join(HERE, "native", "deny_threads.c"), "-ldl"],
                   check=True)
    r = subprocess.run([sys.executable, "-c", SCRIPT.format(root=os.path.dirname(HERE), tests=HERE, shim=shim)],
                       env=dict(os.environ, LD_PRELOAD=shim), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert int(r.stdout.split()[-1]) >= 7, r.stdout  # six schedules, and the ensemble's workers


def test_schedules_of_middling_patterns_are_planned_apart(tmp_path):
    """Patterns of more than 5,000 entries plan their six schedules on host
    threads (asked for here, and denied): one after the other, those of
    scattered columns made a first set-up three times as long."""
    shim = str(tmp_path / "deny_threads.so")
    subprocess.run(["gcc", "-shared", "-fPIC", "-o", shim, os.path.join(HERE, "native", "deny_threads.c"), "-ldl"],
                   check=True)
    script = SCRIPT[:SCRIPT.index("ctx = ")] + r"""
ctx = api.Context(0)
for dims in ((12, 10, 5), (30, 30, 1), (4, 4, 4)):
    rp, col = grid(*dims)
    A = api.CompRowMatrix(ctx, len(rp) - 1, rp, col, values(rp, col, 1))
    s = api.BiCGstab(ctx, abi.PC_ILU)
    before = threads.threads_denied()
    threads.deny_threads(1)
    s.set_matrix(A)
    threads.deny_threads(0)
    print(len(col), threads.threads_denied() - before)
"""
    r = subprocess.run([sys.executable, "-c", script.format(root=os.path.dirname(HERE), tests=HERE, shim=shim)],
                       env=dict(os.environ, LD_PRELOAD=shim), capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    got = [tuple(int(v) for v in line.split()) for line in r.stdout.splitlines()]
    assert len(got) == 3 and all(denied == (6 if entries > 5000 else 0) for entries, denied in got), got
