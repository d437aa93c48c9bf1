"""The fused minibatch step of PPO's update (csrc/update_tc.cu) gives the separate kernels' results bit for bit: an update
against the same 16 steps made of Trainer.minibatch (the separate forward, loss and backward) and Adam in FP32 numpy,
which the kernels' arithmetic is (no fused multiply-adds). Only the FP64 sums (log-std gradients, gradient norm, KL) are
added in other orders; they are within 2^-40 of one another and rounded to FP32."""
import ctypes

import numpy as np
import pytest

import warporacer3d_gb300 as W

pytestmark = pytest.mark.gpu

f32 = np.float32
powf = ctypes.CDLL("libm.so.6").powf
powf.restype, powf.argtypes = ctypes.c_float, [ctypes.c_float, ctypes.c_float]


def bits(a):
    return np.ascontiguousarray(a, f32).view(np.uint32)


# inputs of one and two 64-wide blocks and their edges; batches of one sample, less than half a tile, a half tile and one
# sample more, a whole tile, ragged last tiles, ranges of an odd number of 64-sample blocks, more ranges than contexts
@pytest.mark.parametrize("beams,cars,rollout", [(2, 1, 4), (108, 33, 4), (58, 64, 4), (59, 65, 4), (60, 128, 4),
                                                (122, 100, 5), (123, 1024, 16), (108, 2048, 32), (108, 4100, 40),
                                                (108, 4729, 16), (59, 19000, 4)])
def test_update_has_the_separate_kernels_bits(beams, cars, rollout):
    run = W.Runner(W.track("bank"), cars, beams=beams, seed=3, policy_seed=5)
    trainer = W.Trainer(cars, beams=beams, rollout=rollout)
    policy, B = run.policy, trainer.batch
    run.synchronize()
    trainer.rollout(run.sim, policy, run.acts, 0)
    theta0 = policy.theta.numpy()
    kl = trainer.update(policy)
    assert policy.status() == 0
    results = lambda: {**{k: getattr(trainer, k).numpy() for k in ("grad", "d3")},
                       **{k: getattr(trainer.acts, k).numpy() for k in ("h1", "h2", "o")}}
    fused, stats = results(), trainer.stats.numpy()
    fused.update(theta=policy.theta.numpy(), first=trainer.first.numpy(), second=trainer.second.numpy())
    assert np.isfinite(fused["theta"]).all() and not np.array_equal(fused["theta"], theta0)

    mean = stats[1] / f32(4 * B)
    scale = f32(1) / np.sqrt(np.maximum(stats[2] / f32(4 * B) - mean * mean, f32(1e-8)))
    w, first, second = theta0.copy(), np.zeros_like(theta0), np.zeros_like(theta0)
    for k in range(16):
        policy.theta.write(w)
        policy.sync()
        trainer.minibatch(policy, (k % 4 + k // 4) % 4, mean, scale)
        g = trainer.grad.numpy()
        norm = trainer.stats.numpy()[3]
        assert abs(norm - (g.astype(np.float64) ** 2).sum()) <= 2.0 ** -22 * norm
        g = g * np.minimum(f32(1), f32(0.5) / (np.sqrt(norm) + f32(1e-8)))
        first = f32(0.9) * first + f32(0.1) * g
        second = f32(0.999) * second + (f32(0.001) * g) * g
        c1, c2 = f32(1) - f32(powf(0.9, k + 1)), f32(1) - f32(powf(0.999, k + 1))
        w = w - (f32(3e-4) * (first / c1)) / (np.sqrt(second / c2) + f32(1e-5))
        w[-2:] = np.clip(w[-2:], f32(-2), f32(0))
    want = results()
    want.update(theta=w, first=first, second=second)
    for name in ("h1", "h2", "o", "d3", "grad", "first", "second", "theta"):
        assert np.array_equal(bits(fused[name]), bits(want[name])), name
    assert f32(kl) == f32(want["d3"][5].astype(np.float64).sum()) / f32(B)
