"""A lidar shape that the caller sets runs as set: `flat` chooses between a car's beams in warps of their own
(k_lidar_track) and warps across car boundaries (k_lidar_flat) whatever a rule would prefer, the autotuner times both,
and a sim without a shape of its own says which one the rule takes. The kernels that ran are read from the profiler."""
import pytest
import torch

import warporacer3d_gb300 as W

pytestmark = pytest.mark.gpu


def lidar_kernels(call):
    from torch.profiler import ProfilerActivity, profile
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        call()
        torch.cuda.synchronize()
    return {k for e in prof.events() for k in ("k_lidar_track", "k_lidar_flat", "k_lidar_dynamic", "k_lidar_segments")
            if k in e.name}


@pytest.fixture(scope="module", autouse=True)
def profiler():
    for _ in range(2):  # the first profile of a process records nothing
        lidar_kernels(lambda: torch.zeros(1, device="cuda"))


def step_of(sim):
    sim.reset()
    return lambda: sim.step(sim.actions, sim.reward, sim.done, sim.obs)


@pytest.mark.parametrize("beams", [96, 108])  # a car's last warp full, and 12 lanes of it in use
@pytest.mark.parametrize("cars", [1, 77])
@pytest.mark.parametrize("name", ["bank", "bridge"])  # one and two layers
def test_flat_is_as_set(name, cars, beams):
    sim = W.Sim(W.track(name), cars, 9, beams=beams)
    step = step_of(sim)
    for cars_per_block, wide in ((2, 0), (4, 1), (8, 0)):
        for flat, kernel in ((0, "k_lidar_track"), (1, "k_lidar_flat"), (0, "k_lidar_track")):
            sim.set_lidar_shape(cars_per_block, wide, flat=flat)
            assert sim.lidar_shape()["flat"] == flat
            assert lidar_kernels(step) == {kernel}, (cars_per_block, wide, flat)
    sim.set_lidar_shape(2, dynamic=1)
    assert sim.lidar_shape()["flat"] == 0 and lidar_kernels(step) == {"k_lidar_dynamic"}


@pytest.mark.parametrize("cars,beams", [(77, 96), (77, 108), (300, 1081)])
def test_shape_read_back_is_what_runs(cars, beams):
    sim = W.Sim(W.track("bridge"), cars, 9, beams=beams)
    ran = lidar_kernels(step_of(sim))
    shape = sim.lidar_shape()
    assert ran == {"k_lidar_flat" if shape["flat"] else "k_lidar_track"}
    sim.set_lidar_shape(shape["cars_per_block"], shape["wide"], shape["split"], None, shape["dynamic"], shape["flat"])
    assert sim.lidar_shape() == shape and lidar_kernels(step_of(sim)) == ran


def test_autotuner_times_both():
    sim = W.Sim(W.track("bank"), 64, 9, beams=108)
    sim.reset()
    sim.reward.numpy()
    assert {"k_lidar_track", "k_lidar_flat", "k_lidar_dynamic"} <= lidar_kernels(lambda: sim.autotune(1))


def test_split_segments_take_the_choice():
    tracks = [W.track("flat"), W.track("bridge")]
    sim = W.Sim.segments(tracks, [40, 33], [1, 2], beams=108)
    step = step_of(sim)
    for flat, kernel in ((0, "k_lidar_track"), (1, "k_lidar_flat")):
        sim.set_lidar_shape(2, split=1, flat=flat)
        assert sim.lidar_shape()["flat"] == flat and lidar_kernels(step) == {kernel}
    sim.set_lidar_shape(2)
    assert lidar_kernels(step) == {"k_lidar_segments"}


@pytest.mark.parametrize("flat", [-1, 2])
def test_other_values_are_refused(flat):
    sim = W.Sim(W.track("bank"), 4, 9)
    with pytest.raises(W.RacerError):
        sim.set_lidar_shape(2, flat=flat)


def test_the_rule_without_a_choice():
    """k_lidar_flat from 2^13 blocks of two cars' own warps on, where a car's last warp would idle lanes; a rollout's
    chains go by the whole sim; launches of one segment of several keep a car's beams together."""
    track = W.track("bank")
    for cars, beams, flat in ((4094, 108, 0), (4095, 108, 1), (4096, 96, 0), (6000, 96, 0), (480, 1081, 0),
                              (481, 1081, 1), (482, 1081, 1)):
        sim = W.Sim(track, cars, 9, beams=beams)
        assert sim.lidar_shape()["flat"] == flat
        assert lidar_kernels(step_of(sim)) == {"k_lidar_flat" if flat else "k_lidar_track"}, (cars, beams)
    run = W.Runner(track, 4096, beams=108)
    run.sim.set_chains(4)
    run.rollout(2)
    run.synchronize()
    assert lidar_kernels(lambda: (run.rollout(2), run.synchronize())) == {"k_lidar_flat"}


def test_segments_keep_a_cars_beams_together():
    tracks = [W.track(name) for name in ("flat", "bridge", "bank", "ramp")]
    sim = W.Sim.segments(tracks, [1, 9000, 5423, 997], [1, 2, 3, 4], beams=1081)  # 7712 x 34 blocks: a launch a segment
    assert sim.lidar_shape()["flat"] == 0
    assert lidar_kernels(step_of(sim)) == {"k_lidar_track"}
