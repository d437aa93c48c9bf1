"""Where the lidar's launch changes with the size: warps across car boundaries where a car's last warp would leave
lanes idle, against the oracle; and a launch a segment in place of the segment table from 2^18
blocks on, against the table (the same cars with more of them to a block), a segment of one car among them."""
import numpy as np
import pytest

import oracle as O
import warporacer3d_gb300 as W

pytestmark = pytest.mark.gpu


def same(a, b):
    return np.array_equal(np.ascontiguousarray(a).view(np.uint32), np.ascontiguousarray(b).view(np.uint32))


@pytest.mark.parametrize("beams", [2, 29, 30, 33, 58, 59, 96, 108])
@pytest.mark.parametrize("name,n", [("bridge", 37), ("bank", 1)])
def test_ragged_beams_equal_oracle(name, n, beams):
    track = W.track(name)
    gpu, cpu = W.Sim(track, n, 9, beams=beams), O.Sim(track, n, 9, beams=beams)
    gpu.reset()
    cpu.reset()
    act = np.random.default_rng(beams).uniform(-1, 1, (2, n)).astype(np.float32)
    for _ in range(3):
        gpu.actions.write(act)
        cpu.actions[:] = act
        gpu.step(gpu.actions, gpu.reward, gpu.done, gpu.obs)
        cpu.step(cpu.actions, cpu.reward, cpu.done, cpu.obs)
        assert same(gpu.obs.numpy(), cpu.obs) and same(gpu.state.numpy(), cpu.state)


def test_launch_a_segment_equals_the_table():
    tracks = [W.track(name) for name in ("flat", "bridge", "bank", "ramp")]
    cars = [1, 9000, 5423, 997]  # 7712 x 34 blocks of 2 cars: past 2^18; a quarter of that at 8 cars a block
    sims = [W.Sim.segments(tracks, cars, [1, 2, 3, 4], beams=1081) for _ in range(2)]
    sims[0].set_lidar_shape(2, 0, 0, [2, 0, 3, 1])
    sims[1].set_lidar_shape(8, 0, 0, None)
    act = np.random.default_rng(1).uniform(-1, 1, (2, sum(cars))).astype(np.float32)
    for sim in sims:
        sim.reset()
        sim.actions.write(act)
    for _ in range(2):
        for sim in sims:
            sim.step(sim.actions, sim.reward, sim.done, sim.obs)
        assert same(sims[0].obs.numpy(), sims[1].obs.numpy()) and same(sims[0].state.numpy(), sims[1].state.numpy())
