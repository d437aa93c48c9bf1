"""The fused minibatch step of PPO's update (csrc/update_tc.cu) against the separate kernels it replaces.

`Trainer.minibatch` runs forward, loss and backward as separate launches on the same theta and rollout, so one update's
last minibatch can be repeated from the state the fused update left: with theta put back to what the last minibatch
saw, activations and loss derivatives must have the same bits, and the gradient may differ only by the order its sums
add in: each of the two adds at most 896-term FP32 chains (2^-24 relative a term) and at most 304 partial sums, so
within 2 * (896 + 304) * 2^-24 of the sum of the terms' magnitudes; that sum is taken from FP64 products."""
import numpy as np
import pytest

import warporacer3d_gb300 as W

pytestmark = pytest.mark.gpu

ORDER = 2 * (896 + 304) * 2.0 ** -24


def setup(beams, cars, rollout):
    run = W.Runner(W.track("bank"), cars, beams=beams, seed=3, policy_seed=5)
    trainer = W.Trainer(cars, beams=beams, rollout=rollout)
    run.synchronize()
    trainer.rollout(run.sim, run.policy, run.acts, 0)
    return run, trainer


# inputs of one and two 64-wide blocks, the widest (128) and the last narrower one; batches of a few samples, a whole
# tile, a ragged last tile, fewer tiles than SMs, more tiles than both contexts of every SM
@pytest.mark.parametrize("beams,cars,rollout", [(2, 1, 4), (58, 128, 4), (59, 100, 5), (60, 33, 4), (123, 1024, 16),
                                                (108, 4100, 40), (122, 513, 8)])
def test_last_minibatch_repeats(beams, cars, rollout):
    run, trainer = setup(beams, cars, rollout)
    policy, B = run.policy, trainer.batch
    before = policy.theta.numpy().astype(np.float64)
    trainer.update(policy)
    assert policy.status() == 0
    after = policy.theta.numpy()
    assert np.isfinite(after).all() and not np.array_equal(after, before.astype(np.float32))
    fused = {k: getattr(trainer, k).numpy() for k in ("grad", "d3", "stats")}
    fused.update({k: getattr(trainer.acts, k).numpy() for k in ("h1", "h2", "o")})
    # theta before the last Adam step, from its moments and gradient (racer/ppo.mojo:317-337 run backwards in FP32)
    f32 = np.float32
    first, second, stats = trainer.first.numpy(), trainer.second.numpy(), fused["stats"]
    c1, c2 = f32(1) - f32(0.9) ** f32(16), f32(1) - f32(0.999) ** f32(16)
    step = (f32(3e-4) * (first / c1)) / (np.sqrt(second / c2) + f32(1e-5))
    policy.theta.write(after + step)
    policy.sync()
    mean = stats[1] / f32(4 * B)
    var = stats[2] / f32(4 * B) - mean * mean
    trainer.minibatch(policy, 2, mean, f32(1) / np.sqrt(max(var, f32(1e-8))))  # (epoch 3, minibatch 3) is minibatch 2
    # theta differs by its own rounding (2^-24 relative) from the one the last minibatch saw, so a few of the BF16
    # operands round the other way: one weight in 2^8 of them at most by 2^-8 of itself
    h1, h2, o = (getattr(trainer.acts, k).numpy() for k in ("h1", "h2", "o"))
    for a, b in ((fused["h1"], h1), (fused["h2"], h2), (fused["o"], o), (fused["d3"], trainer.d3.numpy())):
        assert np.linalg.norm(a - b) <= 2.0 ** -8 * np.linalg.norm(b)
    g, ref = fused["grad"], trainer.grad.numpy()
    assert np.linalg.norm(g - ref) <= 2.0 ** -7 * np.linalg.norm(ref)
    # the gradient of the fused kernel's own operands in FP64: its products round to BF16 what the separate ones do
    def bf16(v):
        u = np.ascontiguousarray(v, np.float32).view(np.uint32)
        return ((u + 0x7FFF + ((u >> 16) & 1)) & 0xFFFF0000).astype(np.uint32).view(np.float32).astype(np.float64)
    d3, h2f = fused["d3"][:3], fused["h2"]
    lay = {"W2": (policy.W2, policy.LOGSTD)}
    terms, mags = bf16(d3) @ bf16(h2f).T, np.abs(bf16(d3)) @ np.abs(bf16(h2f)).T
    lo, hi = lay["W2"]
    assert np.all(np.abs(g[lo:hi] - terms.ravel()) <= ORDER * mags.ravel() + 1e-30)
    want = fused["d3"][3:5].astype(np.float64).sum(1)
    assert np.all(np.abs(g[policy.LOGSTD:] - want) <= 2.0 ** -23 * np.abs(fused["d3"][3:5]).astype(np.float64).sum(1))


@pytest.mark.parametrize("beams,cars,rollout", [(108, 2048, 32), (59, 100, 5)])
def test_update_matches_the_separate_kernels(beams, cars, rollout):
    """A whole update (16 dependent minibatches) against the same steps made from Trainer.minibatch and Adam in numpy:
    theta within 2^-10 of its change, the size of a BF16 rounding that goes the other way in a few weights."""
    run, trainer = setup(beams, cars, rollout)
    policy, B = run.policy, trainer.batch
    theta0 = policy.theta.numpy()
    kl = trainer.update(policy)
    theta = policy.theta.numpy()
    f32 = np.float32
    stats = trainer.stats.numpy()
    mean = stats[1] / f32(4 * B)
    scale = f32(1) / np.sqrt(max(stats[2] / f32(4 * B) - mean * mean, f32(1e-8)))
    policy.theta.write(theta0)
    policy.sync()
    w, first, second = theta0.copy(), np.zeros_like(theta0), np.zeros_like(theta0)
    for k in range(16):
        trainer.minibatch(policy, (k % 4 + k // 4) % 4, mean, scale)
        g = trainer.grad.numpy()
        norm = f32((g.astype(np.float64) ** 2).sum())
        g = g * min(f32(1), f32(0.5) / (np.sqrt(norm) + f32(1e-8)))
        first = f32(0.9) * first + f32(0.1) * g
        second = f32(0.999) * second + (f32(0.001) * g) * g
        t = f32(k + 1)
        c1, c2 = f32(1) - f32(0.9) ** t, f32(1) - f32(0.999) ** t
        w = w - (f32(3e-4) * (first / c1)) / (np.sqrt(second / c2) + f32(1e-5))
        w[-2:] = np.clip(w[-2:], -2, 0)
        policy.theta.write(w)
        policy.sync()
    change = np.linalg.norm(w - theta0)
    assert np.linalg.norm(theta - w) <= 2.0 ** -10 * change
    assert abs(kl - trainer.d3.numpy()[5].astype(np.float64).mean()) <= 2.0 ** -10 * max(abs(kl), 1e-6)
