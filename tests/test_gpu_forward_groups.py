"""The register-staged BF16 forward with two and with four k-blocks in flight, which share two stages: which one runs
(read from the profiler) at the sizes where they take over from one another, with as many k-blocks as leave a group
without work, its first, or a second use of a stage, and that they give the same bits for the same samples. The sizes
follow the device's SM count."""
import numpy as np
import pytest
import torch

import warporacer3d_gb300 as W

pytestmark = pytest.mark.gpu

SAMPLES = 128  # a tile's


def kernels(call):
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        call()
        torch.cuda.synchronize()
    return {k for e in prof.events() for k in ("k_mlp_fwd<2>", "k_mlp_fwd<4>", "k_mlp_fwd_tma") if k in e.name}


@pytest.fixture(scope="module", autouse=True)
def profiler():
    for _ in range(2):  # the first profile of a process records nothing
        kernels(lambda: torch.zeros(1, device="cuda"))


def bits(a):
    return np.ascontiguousarray(a).view(np.uint32)


# inputs of 2, 3, 4, 5, 6, 8, 9, 10, 11 and 17 k-blocks
@pytest.mark.parametrize("inputs", [128, 129, 256, 257, 321, 512, 513, 640, 641, 1086])
def test_groups(inputs):
    sms, kb = torch.cuda.get_device_properties(0).multi_processor_count, (inputs + 63) // 64
    policy = W.Policy(3, beams=inputs - 5)
    most = sms * SAMPLES + 4
    x = np.random.default_rng(inputs).uniform(-1, 1, (inputs, most)).astype(np.float32)
    whole = None
    for cols in (most, most - 4, most - 5, sms // 2 * SAMPLES + 1, sms // 2 * SAMPLES, 8 * SAMPLES + 1, 8 * SAMPLES, 129, 1):
        xd = W.DevArray.empty((inputs, cols))
        xd.write(np.ascontiguousarray(x[:, :cols]))
        acts = W.Activations(policy, cols)
        ran = kernels(lambda: policy.forward(xd, acts))
        tiles = (cols + SAMPLES - 1) // SAMPLES
        want = ("k_mlp_fwd_tma" if kb > 4 and tiles > sms and cols % 4 == 0 else
                "k_mlp_fwd<4>" if kb > 2 and (tiles <= 8 or kb > 10 and 2 * tiles <= sms) else "k_mlp_fwd<2>")
        assert ran == {want}, (cols, ran)
        got = {name: getattr(acts, name).numpy() for name in ("h1", "h2", "o")}
        whole = whole or got
        for name in got:
            assert np.array_equal(bits(got[name]), bits(whole[name][:, :cols])), (name, cols)
    assert policy.status() == 0


def test_a_chains_part_takes_two():
    """A chain steps its cars beside the other chains' lidars: two k-blocks in flight, and the one-chain rollout's bits."""
    runs = [W.Runner(W.track("bridge"), 2048, beams=1081, seed=3, policy_seed=5) for _ in range(2)]
    runs[1].sim.set_chains(4)
    for run, kernel in zip(runs, ("k_mlp_fwd<4>", "k_mlp_fwd<2>")):
        for t in (0, 4):
            run.rollout(4, False, t)
            run.synchronize()
        assert kernels(lambda: (run.rollout(4, False, 8), run.synchronize())) == {kernel}
    for key in ("obs", "state", "actions"):
        a, b = (getattr(run.sim, key).numpy() for run in runs)
        assert np.array_equal(bits(a), bits(b)), key
