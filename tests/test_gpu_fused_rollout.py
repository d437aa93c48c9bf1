"""The fused rollout where its forward changes: inputs that just fill one k-block, two, and spill into the next (64 and
128 inputs are beams of 59 and 123), with one car a CTA, a few, and more than the 32 rows that a CTA's staging passes
take at a time, against the chained graph, bit for bit."""
import numpy as np
import pytest

import warporacer3d_gb300 as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("beams", [59, 60, 123, 124])
@pytest.mark.parametrize("n", [3, 1205, 10500])
def test_fused_rollout_at_input_edges(n, beams):
    track = W.track("bank")
    chained = W.Runner(track, n, beams=beams, seed=13, policy_seed=5)
    fused = W.Runner(track, n, beams=beams, seed=13, policy_seed=5)
    fused.sim.set_fused_rollout(True)
    for runner in (chained, fused):
        runner.rollout(5, False, 40)
        runner.rollout(5, False, 45)  # starts from observations that the first launch left
        runner.synchronize()
    for arr in ("state", "obs", "actions", "reward", "done"):
        a, b = getattr(chained.sim, arr).numpy(), getattr(fused.sim, arr).numpy()
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32)), arr
    assert fused.policy.status() == 0
