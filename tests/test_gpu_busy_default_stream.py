"""Objects made on a caller's non-blocking stream while the default stream is busy: their memory is zeroed before the
call returns, not behind the default stream's work, where it would wipe what their own stream's first kernels wrote."""
import numpy as np
import pytest

import warporacer3d_gb300 as W

pytestmark = pytest.mark.gpu


def results(stream, busy):
    import torch
    rng = np.random.default_rng(1)

    def hold():  # about a tenth of a second of default-stream work ahead of what follows
        if busy:
            torch.cuda._sleep(200_000_000)
    out = {}
    hold()
    policy = W.Policy(5, beams=108, stream=stream)
    out["theta"] = policy.theta.numpy()
    cols = 1000
    x = W.DevArray.empty((113, cols))
    x.write(rng.uniform(-1, 1, (113, cols)))
    d3 = W.DevArray.empty((3, cols))
    d3.write(rng.uniform(-1, 1, (3, cols)))
    d2, d1, grad = W.DevArray.empty((65, cols)), W.DevArray.empty((65, cols)), W.DevArray.empty((policy.P,))
    hold()
    acts = W.Activations(policy, cols)
    policy.forward(x, acts)
    policy.sync()
    hold()
    policy.backward(x, acts, d3, d2, d1, grad)
    policy.status()
    out["grad"] = grad.numpy()[:policy.LOGSTD]
    sim = W.Sim(W.track("bank"), 32, 3, beams=108, stream=stream)
    sim.reset()
    hold()
    net = W.Surrogate(sim, hidden=128, batch=1024, seed=3)
    net.set_poses(1024, 7)
    out["net"] = net.theta.numpy()
    hold()
    out["mse"] = np.float32(net.gradient(0))
    trainer = W.Trainer(32, beams=108, rollout=8, stream=stream)
    run = W.Runner(None, None, beams=108, sim=sim, policy_seed=5)
    hold()
    trainer.rollout(sim, run.policy, run.acts, 0)
    trainer.update(run.policy)
    out["trained"] = run.policy.theta.numpy()
    hold()
    out["snapshot"] = sim.snapshot()
    hold()
    out["evaluated"] = np.array(run.evaluate_graph(8))
    hold()
    run.rollout_surrogate(net, 4, True, 0, 2, 0.5)
    out["obs"] = sim.obs.numpy()
    torch.cuda.synchronize()
    return out


def test_busy_default_stream():
    import torch
    stream = torch.cuda.Stream()
    idle, busy = results(stream, False), results(stream, True)
    for key in ("theta", "grad", "net", "trained", "snapshot", "evaluated", "obs"):
        assert np.any(idle[key]) and np.array_equal(idle[key], busy[key]), key
    assert idle["mse"] > 0 and abs(idle["mse"] - busy["mse"]) <= 2.0 ** -20 * idle["mse"]  # its terms are added by atomics
