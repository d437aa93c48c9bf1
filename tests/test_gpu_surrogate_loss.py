"""The learned lidar's loss sums: a squared error past FP32's largest value is an infinite loss (not a NaN), and the mean
of equal errors is that error's square to FP32's rounding of the terms."""
import numpy as np
import pytest

import warporacer3d_gb300 as W

pytestmark = pytest.mark.gpu


def net_with_outputs(frame, beams, value, batch=1024):
    """A surrogate whose every output is `value` (a bias beside which the rest vanishes) and a buffer for its labels."""
    sim = W.Sim(W.track("bridge"), 8, 7, beams=beams)
    sim.reset()
    net = W.Surrogate(sim, hidden=256, batch=batch, seed=3, frame=frame)
    net.set_poses(batch, 11)
    theta, (off, shape) = net.theta.numpy(), net.layout()["b4"]
    theta[off:off + shape[0]] = value
    net.theta.write(theta)
    return net, W.DevArray.empty((beams, batch))


@pytest.mark.parametrize("frame,beams", [("car", 108), ("car_grid", 109), ("world", 1081)])
def test_overflowing_loss_is_infinite(frame, beams):
    net, labels = net_with_outputs(frame, beams, 1e25)
    assert net.gradient(0, labels) == np.inf


@pytest.mark.parametrize("frame,beams", [("car", 108), ("car_grid", 109), ("world", 1081)])
def test_loss_is_the_mean_square(frame, beams):
    net, labels = net_with_outputs(frame, beams, 1e15)
    mse = net.gradient(0, labels)
    want = np.mean((np.float64(np.float32(1e15)) - labels.numpy().astype(np.float64)) ** 2)
    # the output, the error and its square, rounded in FP32, and 16 of them summed in FP32; then the result's rounding
    assert abs(mse - want) <= (2 + 1 + 16 + 1) * 2.0 ** -24 * want
