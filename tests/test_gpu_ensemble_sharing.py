"""rsg_ensemble_step_batched: a member's result does not depend on the members
listed with it, on their order or on who shares its context, on either route
(streams of their own, or lockstep)."""
import os
import subprocess
import sys

import numpy as np
import pytest

from ressim_gb300 import abi, api
from ressim_gb300 import workloads as W

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
SIZES = [(33, 34, 5), (16, 16, 6), (20, 8, 3)]


def member(ctx, k, **kw):
    return W.build_two_phase_sim(ctx, *SIZES[k], seed=70 + k, rtol=1e-10, stop_rule=1, **kw)


def stepped(order, ctx_of, precision, bystanders=()):
    """The states of the members `order` after two steps of the call; member k
    lives on context number ctx_of[k]."""
    ctxs = {c: api.Context(0) for c in set(ctx_of.values())}
    try:
        others = [member(ctxs[ctx_of[k]], k) for k in bystanders]
        sims = [member(ctxs[ctx_of[k]], k) for k in order]
        for _ in range(2):
            _, sts = api.ensemble_step_batched([s for s, _ in sims], [c["dt"] for _, c in sims], precision=precision)
            assert not sts.any(), sts
        out = {k: s.state() for k, (s, _) in zip(order, sims)}
        del others
        return out
    finally:
        for c in ctxs.values():
            c.close()


@pytest.mark.parametrize("precision", [0, 1])
def test_same_bits_whoever_is_listed(precision):
    alone = {k: stepped([k], {k: 0}, precision)[k] for k in range(3)}
    runs = [stepped([0, 1, 2], {0: 0, 1: 0, 2: 0}, precision),
            stepped([2, 1, 0], {0: 0, 1: 0, 2: 1}, precision),
            stepped([0], {0: 0, 1: 0}, precision, bystanders=[1])]
    for r in runs:
        for k, state in r.items():
            for got, want in zip(state, alone[k]):
                assert np.array_equal(got, want), k


def test_shared_context_is_itself_again(ctx):
    """Members on one context, one of them failing and one with a solver that
    ensembles do not take: the others step, the context holds the failure's
    message and counts every launch, and its simulators go on as alone."""
    one = api.Context(0)
    alone = api.Context(0)
    try:
        sims = [member(one, k) for k in range(3)]
        other, case = member(one, 1, method=abi.GMRES)
        dts = [c["dt"] for _, c in sims]
        before = one.kernel_launches()
        _, sts = api.ensemble_step_batched([s for s, _ in sims] + [other], [-1.0] + dts[1:] + [case["dt"]])
        assert sts[0] == abi.BAD_ARG and not sts[1:3].any() and sts[3] == abi.UNSUPPORTED
        assert one.kernel_launches() - before > 20
        assert "positive" in api.lib().rsg_context_last_error(one.h).decode()
        one.set_profiling(True)
        one.profile_reset()
        _, sts = api.ensemble_step_batched([sims[1][0], sims[2][0]], dts[1:])
        assert not sts.any()
        assert one.profile()["assemble_rows"][1] >= 4
        one.set_profiling(False)
        sims[1][0].step(dts[1])
        ref, _ = member(alone, 1)
        for _ in range(2):
            api.ensemble_step_batched([ref], dts[1:2])
        ref.step(dts[1])
        for got, want in zip(sims[1][0].state(), ref.state()):
            assert np.array_equal(got, want)
    finally:
        one.close()
        alone.close()


def test_lockstep_members():
    """The batched tests once more without block walks: members begin on their
    own streams and go on in lockstep, as those do whose pattern or factors
    have none."""
    r = subprocess.run([sys.executable, "-m", "pytest", "-x", "-q", os.path.join(HERE, "test_gpu_ensemble.py"),
                        os.path.join(HERE, "test_gpu_ensemble_routes.py"),
                        os.path.join(HERE, "test_gpu_ensemble_sharing.py"), "-k",
                        "batched_ensemble or routes_agree or same_bits or itself_again"],
                       env=dict(os.environ, RSG_SWEEP="ring"), capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-1000:]
    assert "13 passed" in r.stdout, r.stdout
