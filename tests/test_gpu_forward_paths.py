"""The BF16 policy forward's paths give the same bits for the same samples: four producer groups (more than 128 inputs
and at most 1024 samples), two groups, and the persistent TMA-staged kernel (more than 256 inputs, more tiles of 128
samples than SMs, sample columns of a multiple of four), at and beside the sizes where one takes over from another."""
import numpy as np
import pytest

import warporacer3d_gb300 as W

pytestmark = pytest.mark.gpu


def same(a, b):
    return np.array_equal(np.ascontiguousarray(a).view(np.uint32), np.ascontiguousarray(b).view(np.uint32))


@pytest.mark.parametrize("beams", [123, 124, 251, 252, 1081])
def test_forward_paths_agree(beams):
    policy = W.Policy(3, beams=beams)
    most = 152 * 128 + 132  # two tiles and a bit past one per SM
    x = np.random.default_rng(beams).uniform(-1, 1, (beams + 5, most)).astype(np.float32)
    ref = None
    for cols in (1, 127, 1024, 1025, 152 * 128, most - 1, most):
        xd = W.DevArray.empty((beams + 5, cols))
        xd.write(np.ascontiguousarray(x[:, :cols]))
        acts = W.Activations(policy, cols)
        policy.forward(xd, acts)
        got = {name: getattr(acts, name).numpy() for name in ("h1", "h2", "o")}
        if ref is not None:  # the shorter batch's samples are the longer's first
            for name in got:
                assert same(got[name][:, :ref[name].shape[1]], ref[name]), (name, cols)
        ref = got
    assert policy.status() == 0
