"""Kernels launched before the one they follow has ended (common.cuh, launch_early) read what that one writes through
the coherent path: the read-only path (ld.global.nc, from __ldg or const __restrict__) requires memory that nothing
writes while the kernel is resident. The sources are checked on the CPU. On the GPU, calls queued one behind another
without a wait give the bits of the same calls with a wait after each: sizes of a few blocks, of less than a wave and
of many."""
import re
from pathlib import Path

import numpy as np
import pytest

import warporacer3d_gb300 as W

CSRC = Path(__file__).resolve().parent.parent / "warporacer3d_gb300" / "csrc"
# what no kernel writes: the track (t., its cells by p, hp and the nearest-waypoint grid) and the beam table
UNWRITTEN = r"(?:reinterpret_cast<[^()]*>\()?(?:t\.|p\b|hp\b|beam_dir\b)"


def kernels(text):
    """(signature, body) of every __global__ function."""
    for m in re.finditer(r"__global__", text):
        depth, k = 0, text.index("{", m.start())
        for end in range(k, len(text)):
            depth += {"{": 1, "}": -1}.get(text[end], 0)
            if depth == 0:
                break
        yield text[m.start():k], text[k:end]


@pytest.mark.parametrize("unit", ["sim.cu", "mlp_tc.cu", "update_tc.cu", "surrogate.cu", "gemm_tc.cuh"])
def test_early_kernels_load_coherently(unit):
    text = re.sub(r"//[^\n]*", "", (CSRC / unit).read_text())
    early = [(s, b) for s, b in kernels(text) if re.search(r"\bearly_(wait|start)\(", b)]
    assert early
    for signature, body in early:
        read_only = re.findall(r"const [\w:]+\s*\*\s*__restrict__\s+(\w+)", signature)
        assert set(read_only) <= {"beam_dir"}, signature
        assert not re.findall(r"__ldg\((?!" + UNWRITTEN + ")[^\n]*", body), signature


@pytest.mark.parametrize("unit,functions", [("sim.cu", ["trace", "beam_range", "trace_any"])])
def test_functions_of_early_kernels_load_coherently(unit, functions):
    text = re.sub(r"//[^\n]*", "", (CSRC / unit).read_text())
    for name in functions:
        found = re.findall(r"\b" + name + r"\((const TrackDev& t[^)]*)\)\s*\{(.*?)\n\}", text, re.S)
        assert found, name
        for signature, body in found:
            assert set(re.findall(r"__restrict__\s+(\w+)", signature)) <= {"beam_dir"}, name
            assert not re.findall(r"__ldg\((?!" + UNWRITTEN + ")[^\n]*", body), name


@pytest.mark.parametrize("unit", ["surrogate.cu", "gemm_epi.cuh", "fwd_tc.cuh", "sample.cuh", "loss.cuh"])
def test_epilogues_of_early_kernels_load_coherently(unit):
    assert "__ldg(" not in re.sub(r"//[^\n]*", "", (CSRC / unit).read_text())


def bits(a):
    return np.ascontiguousarray(a).view(np.uint32)


@pytest.mark.gpu
@pytest.mark.parametrize("name,cars,beams", [("bank", 16, 108), ("bridge", 64, 108), ("bridge", 2999, 271),
                                             ("bridge", 4096, 1081), ("bank", 20000, 108)])
def test_queued_sim_steps(name, cars, beams):
    steps, track = 32, W.track(name)
    acts = np.random.default_rng(cars).uniform(-1, 1, (steps, 2, cars)).astype(np.float32)
    sims = [W.Sim(track, cars, 7, beams=beams) for _ in range(2)]
    given = W.DevArray.empty(acts.shape)
    given.write(acts)
    for sim, wait in zip(sims, (False, True)):
        sim.reset()
        sim.reward.numpy()
        for k in range(steps):
            sim.step(given[k], sim.reward, sim.done, sim.obs)
            if wait:
                sim.reward.numpy()
    for key in ("obs", "state", "reward", "done"):
        a, b = (getattr(sim, key).numpy() for sim in sims)
        assert np.array_equal(bits(a), bits(b)), key


@pytest.mark.gpu
@pytest.mark.parametrize("cars,beams", [(16, 108), (2999, 271), (4096, 1081), (30000, 271)])
def test_queued_runner_steps(cars, beams):
    runs = [W.Runner(W.track("bridge"), cars, beams=beams, seed=3, policy_seed=5) for _ in range(2)]
    for run, wait in zip(runs, (False, True)):
        run.synchronize()
        for t in range(32):
            run.step(False, t)
            if wait:
                run.synchronize()
        run.synchronize()
    for key in ("obs", "state", "actions", "reward"):
        a, b = (getattr(run.sim, key).numpy() for run in runs)
        assert np.array_equal(bits(a), bits(b)), key
    assert all(run.policy.status() == 0 for run in runs)


@pytest.mark.gpu
@pytest.mark.parametrize("frame,beams", [("car", 108), ("car_grid", 109), ("world", 1081)])
def test_gradients_of_other_batches_before(frame, beams):
    """A training batch's kernels start early behind one another on buffers that the batch before used: the weights'
    gradients, whose sums have a fixed order, have the same bits whatever batches came before."""
    sim = W.Sim(W.track("bridge"), 64, 7, beams=beams)
    sim.reset()
    grads = []
    for order in (range(4), reversed(range(4))):
        net = W.Surrogate(sim, hidden=256, batch=1024, seed=3, frame=frame)
        net.set_poses(4096, 11)
        got = {}
        for again in range(2):  # labels traced, then read in place
            for b in (order if again == 0 else sorted(got)):
                net.gradient(b * 1024)
                grad, blocks = net.grad.numpy(), net.layout()
                got[b] = {w: grad[off:off + int(np.prod(shape))] for w, (off, shape) in blocks.items() if w[0] == "W"}
        grads.append(got)
    for b in range(4):
        for w in ("W1", "W2", "W3", "W4"):
            assert np.any(grads[0][b][w]) and np.array_equal(bits(grads[0][b][w]), bits(grads[1][b][w])), (b, w)
