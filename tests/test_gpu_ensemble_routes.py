"""rsg_ensemble_step_batched: members on their own streams (a context each) and
members stepped in lockstep (contexts shared) in one call, against each member
stepped alone."""
import numpy as np
import pytest

from ressim_gb300 import api
from ressim_gb300 import workloads as W

pytestmark = pytest.mark.gpu

SIZES = [(16, 16, 6), (12, 10, 4), (33, 34, 5), (20, 8, 3)]


@pytest.mark.parametrize("shared", [(), (1, 3), (0, 1, 2, 3)])
@pytest.mark.parametrize("precision", [0, 1])
def test_routes_agree(shared, precision):
    """Linear solves to 1e-12 and the max |dp/p| Newton stop rule (as the
    serial comparison of the FP64 launch): equal Newton counts, pressures
    within 1e-10 of the serial step and 1e-12 mass balance on either route; a
    failing member (a time step below zero) leaves the others alone."""
    one = api.Context(0)
    ctxs = [one if k in shared else api.Context(0) for k in range(len(SIZES))]
    alone = api.Context(0)
    build = lambda c, k: W.build_two_phase_sim(c, *SIZES[k], seed=60 + k, rtol=1e-12, stop_rule=1)  # noqa: E731
    try:
        sims, cases = zip(*[build(c, k) for k, c in enumerate(ctxs)])
        dts = [case["dt"] for case in cases]
        infos, sts = api.ensemble_step_batched(sims, dts, precision=precision)
        assert not sts.any(), sts
        p = [s.state()[0].copy() for s in sims]
        for k in range(len(SIZES)):
            ref, case = build(alone, k)
            i = ref.step(case["dt"])
            assert i.newton_iterations == infos[k].newton_iterations
            assert infos[k].mass_balance_error <= 1e-12
            q = ref.state()[0]
            assert np.max(np.abs(p[k] - q) / np.abs(q)) <= 1e-10
        infos, sts = api.ensemble_step_batched(sims, [-1.0] + dts[1:], precision=precision)
        assert sts[0] != 0 and not sts[1:].any()
    finally:
        for c in {id(c): c for c in ctxs + [one, alone]}.values():
            c.close()
