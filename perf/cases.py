"""The work that a program using this package has it do, as cases to be measured.

A case names a kind of call and its sizes. `prepare` makes what such a program has in hand before the call (a sim
on a track, a policy, rollout storage, a trained lidar's weights), `run` makes one pass through the public entry
points and returns views of everything the pass wrote, `work` counts the bytes and operations the pass cannot do
without, `exact` gives the policy's products in 64 bits.
"""
import functools
import math

import numpy as np
import torch

import warporacer3d_gb300 as W
from warporacer3d_gb300.tracks import compile as track_compile

H, HA, OUT = 64, 65, 3
BATCH_TRACKS = ("flat", "ramp", "bank", "bridge", "occupancy")
BATCH_SHARES = (1024, 4096, 16384, 32768, 65536)
PROBES = {"flat": 6, "ramp": 9, "bank": 9, "bridge": 7, "occupancy": 32}  # probes of a beam, about
PROBE_FLOPS, BEAM_FLOPS, CAR_FLOPS = 25, 60, 6000  # of a probe, a beam's set-up, a car's 16 derivatives


def listed():
    return [
        # a viewer or a driving demo: a handful of cars stepped one call at a time
        dict(name="step_16", kind="step", track="flat", cars=16, beams=108),
        # an evaluation loop of per-step calls at a size that fills neither a warp nor a block
        dict(name="step_2999", kind="step", track="ramp", cars=2999, beams=271),
        # cars on five tracks at once, the largest batch the benchmark runs
        dict(name="step_batch", kind="batch", cars=119808, beams=1081),
        # the headline workload: a graph-replayed rollout of the full lidar
        dict(name="rollout_bridge", kind="rollout", track="bridge", cars=4096, beams=1081, steps=64, chains=16),
        # the reference's own benchmark sizes, as the fused persistent rollout the autotuner picks there (chains 0)
        dict(name="rollout_ramp", kind="rollout", track="ramp", cars=1024, beams=108, steps=100, chains=0),
        # collecting PPO's rollout storage, with GAE
        dict(name="ppo_rollout", kind="ppo_rollout", track="bank", cars=16384, beams=108, rollout=64),
        # PPO's update on that storage: 4 epochs of 4 minibatches
        dict(name="ppo_update", kind="ppo_update", track="bank", cars=16384, beams=108, rollout=64, precision="bf16"),
        # a caller's own training loop: one forward and one backward of the policy at the full lidar
        dict(name="policy_bf16", kind="policy", beams=1081, cols=16384, precision="bf16"),
        # the same in FP32, the precision of comparison runs
        dict(name="policy_fp32", kind="policy", beams=1081, cols=4096, precision="fp32"),
        # the learned lidar serving a rollout, one step of sixteen audited by the exact tracer
        dict(name="learned_rollout", kind="learned_rollout", track="bridge", cars=65536, beams=1081, steps=16,
             frame="world"),
        # one batch of the learned lidar's training: labels, forward, loss and gradient
        dict(name="learned_gradient", kind="learned_gradient", track="bridge", beams=1081, hidden=512, batch=8192,
             frame="world"),
        # a track compiled from its route
        dict(name="track_ribbon", kind="track", shape="eight", cell=0.025, ramps=0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "batch", "rollout", "rollout", "ppo_rollout", "ppo_update", "ppo_update",
                       "policy", "policy", "learned_rollout", "learned_gradient", "track"])
    track = rng.choice(["flat", "ramp", "bank", "bridge"])
    if kind == "step":
        beams = _log_int(rng, 9, 1081)
        return dict(kind=kind, track=track, cars=_log_int(rng, 1, min(65536, 20_000_000 // beams)), beams=beams)
    if kind == "batch":
        return dict(kind=kind, cars=_log_int(rng, 500, 60000), beams=rng.choice([108, 271, 540, 1081]))
    if kind == "rollout":
        beams = _log_int(rng, 27, 1081)
        cars = _log_int(rng, 64, min(16384, 4096 * 1081 // beams))
        return dict(kind=kind, track=track, cars=cars, beams=beams, steps=rng.randint(8, 64),
                    chains=rng.choice([0, 1, 3, 8, 16]))
    if kind in ("ppo_rollout", "ppo_update"):
        beams = rng.choice([54, 108, 108, 181, 271, 1081])
        rollout = rng.choice([16, 32, 32, 64])
        cars = _log_int(rng, 100, min(16384, 16384 * 64 * 108 // (beams * rollout)))
        case = dict(kind=kind, track=track, cars=cars, beams=beams, rollout=rollout)
        if kind == "ppo_rollout":
            return case
        if rng.random() < 0.3:  # the precision of comparison runs, at sizes that cost as much
            return dict(case, cars=max(64, cars // 4), precision="fp32")
        return dict(case, precision="bf16")
    if kind == "policy":
        precision = rng.choice(["bf16", "fp32"])
        return dict(kind=kind, beams=_log_int(rng, 9, 1081), cols=_log_int(rng, 1, 16384 if precision == "fp32" else 65536),
                    precision=precision)
    if kind == "learned_rollout":
        return dict(kind=kind, track=track, cars=_log_int(rng, 500, 32768), beams=12 * rng.randint(9, 90) + 1,
                    steps=rng.randint(4, 16), frame=rng.choice(["world", "world", "car_grid", "car"]))
    if kind == "learned_gradient":
        return dict(kind=kind, track=track, beams=12 * rng.randint(9, 90) + 1, hidden=rng.choice([256, 512, 512]),
                    batch=128 * rng.randint(8, 64), frame=rng.choice(["world", "world", "car_grid", "car"]))
    return dict(kind="track", shape=rng.choice(["eight", "oval", "image"]), cell=round(rng.uniform(0.024, 0.06), 4),
                ramps=rng.randint(0, 8))


class _View:
    """A device array of the package, for torch to wrap without a copy."""

    def __init__(self, array):
        self.array = array
        self.__cuda_array_interface__ = {"shape": array.shape, "typestr": array.dtype.str, "data": (array.ptr, False),
                                         "version": 3}


def _view(array):
    return torch.as_tensor(_View(array), device="cuda")


def _device(values):
    array = W.DevArray.empty(values.shape)
    array.write(values)
    return array


@functools.lru_cache(maxsize=None)
def _track(name):
    return W.track(name)


def _batch_cars(cars):
    cuts = np.round(np.cumsum(BATCH_SHARES) / sum(BATCH_SHARES) * cars).astype(int)
    return [int(c) for c in np.maximum(np.diff(np.concatenate([[0], cuts])), 1)]


def _sim_views(sim):
    return {name: _view(getattr(sim, name)) for name in ("state", "obs", "actions", "reward", "done")}


def _route(case, seed):
    """A closed route, the road's half-width and bank, which vary a little with the seed, and its ramps."""
    rng = np.random.default_rng(seed)
    t = np.linspace(0, 2 * np.pi, 160, endpoint=False)
    if case["shape"] == "eight":
        z = 0.9 * np.clip(np.cos((t - np.pi) * 1.4), 0, 1) ** 2
        route = np.column_stack([7 * np.sin(t), 3.5 * np.sin(2 * t), z])
        half_width, bank = 1.1 * (1 + 0.03 * rng.uniform(-1, 1)), 0
    else:
        route = np.column_stack([6 * np.cos(t), 6 * np.sin(t), 0.7 * (1 - np.cos(2 * t))])
        half_width, bank = 1.3 * (1 + 0.03 * rng.uniform(-1, 1)), 0.25 * (1 + 0.1 * rng.uniform(-1, 1))
    ramps = []
    for k in range(case["ramps"]):
        at = int(rng.integers(160))
        d = route[(at + 1) % 160] - route[at]
        ramps.append({"center": [float(route[at, 0]), float(route[at, 1])], "heading": float(np.arctan2(d[1], d[0])),
                      "length": 1.6, "width": 1.0, "height": 0.25})
    return route, half_width, bank, ramps


def _image(case, seed):
    """A free-space image of a wavy ring, its centreline as (row, col) points, and the map's corner."""
    rng = np.random.default_rng(seed)
    cell = case["cell"]
    size = int(24.0 / cell)
    x0 = y0 = -size * cell / 2
    xs = x0 + cell * np.arange(size)
    gx, gy = np.meshgrid(xs, xs)
    free = np.abs(np.hypot(gx, gy) - (8 + 0.8 * np.sin(3 * np.arctan2(gy, gx)))) < 0.9 * (1 + 0.1 * rng.uniform(-1, 1))
    t = np.linspace(0, 2 * np.pi, int(2 * np.pi * 8 / cell), endpoint=False)
    r = 8 + 0.8 * np.sin(3 * t)
    loop = np.column_stack([(r * np.sin(t) - y0) / cell, (r * np.cos(t) - x0) / cell])
    ramps = _route(dict(case, shape="oval"), seed)[3]
    return free, loop, x0, y0, ramps


def _policy_inputs(case, seed):
    """theta, observations (ranges of 10 m, the constant 1 in the last row) and output gradients."""
    rng = np.random.default_rng(seed)
    n, cols = case["beams"] + 5, case["cols"]
    theta = np.concatenate([
        (rng.standard_normal((H, n)) * math.sqrt(2 / (n - 1))).ravel(), (rng.standard_normal((H, HA)) / 8).ravel(),
        (rng.standard_normal((OUT, HA)) / 8).ravel(), [-0.5, -0.5]]).astype(np.float32)
    x = rng.random((n, cols), dtype=np.float32)
    x[-1] = 1
    d3 = (rng.standard_normal((OUT, cols), dtype=np.float32)) * np.float32(1 / cols)
    return theta, x, d3


def _learned_theta(sur, track, seed):
    """Weights whose predictions rise with the clearance at the car, as a trained lidar's smallest ranges do, so
    that the cars beside a wall are the ones that fall back to the exact tracer."""
    rng = np.random.default_rng(seed)
    theta = np.zeros(sur.theta.shape, np.float32)
    scale = {"W1": 0.3 / 8, "W2": 0.3 / math.sqrt(sur.hidden), "W3": 0.3 / math.sqrt(sur.hidden),
             "W4": 0.02 / math.sqrt(sur.hidden)}
    clear = 16 if sur.frame != "car" else 5  # the input that holds it: grid level 2's first feature, or a constant
    for name, (off, shape) in sur.layout().items():
        v = (rng.standard_normal(shape) * scale.get(name, 0.0)).astype(np.float32)
        if name == "W1":
            v[:, clear] = 1.0
        elif name in ("W2", "W3"):
            v += np.float32(1.6 / sur.hidden)
        elif name == "W4":
            v += np.float32(0.3 / sur.hidden)
        elif name == "b4":
            v[:] = -0.07 if sur.frame != "car" else 0.1
        elif name == "G2":
            nx, ny, cell = int(track[0]), int(track[1]), float(track[4])
            step = sur.grid()[2][2] / cell
            for layer in range(shape[0]):
                grid = track[12 + 3 * layer * nx * ny:][:nx * ny].reshape(ny, nx)
                iy = np.minimum((np.arange(shape[1]) * step).astype(int), ny - 1)
                ix = np.minimum((np.arange(shape[2]) * step).astype(int), nx - 1)
                v[layer, :, :, 0] = np.clip(grid[np.ix_(iy, ix)], 0, 1.5)
        theta[off:off + v.size] = v.ravel()
    return theta


def prepare(case, seed):
    kind = case["kind"]
    if kind == "track":
        if case["shape"] == "image":
            return {"case": case, "image": _image(case, seed)}
        return {"case": case, "route": _route(case, seed)}
    s = {"case": case}
    if kind == "policy":
        theta, x, d3 = _policy_inputs(case, seed)
        p = s["policy"] = W.Policy(1, beams=case["beams"])
        p.theta.write(theta)
        p.sync()
        p.set_precision(case["precision"])
        s["x"], s["d3"] = _device(x), _device(d3)
        s["acts"] = W.Activations(p, case["cols"])
        s["back"] = [W.DevArray.empty((HA, case["cols"])), W.DevArray.empty((HA, case["cols"])), W.DevArray.empty((p.P,))]
        s["out"] = {name: _view(getattr(s["acts"], name)) for name in ("h1", "h2", "o")}
        s["out"].update({name: _view(a) for name, a in zip(("d2", "d1", "grad"), s["back"])})
        return s
    if kind == "batch":
        cars = _batch_cars(case["cars"])
        r = W.Runner.segments([_track(t) for t in BATCH_TRACKS], cars, [seed + k for k in range(5)],
                              beams=case["beams"], policy_seed=seed)
    elif kind == "learned_gradient":
        sim = s["sim"] = W.Sim(_track(case["track"]), 128, seed, beams=case["beams"])
        sur = s["sur"] = W.Surrogate(sim, hidden=case["hidden"], batch=case["batch"], seed=seed, frame=case["frame"])
        sur.set_loss(0.02)
        sur.set_poses(case["batch"], seed=seed)
        s["labels"] = W.DevArray.empty((case["beams"], case["batch"]))
        s["out"] = {"grad": _view(sur.grad), "labels": _view(s["labels"])}
        return s
    else:
        r = W.Runner(_track(case["track"]), case["cars"], beams=case["beams"], seed=seed, policy_seed=seed)
    s["runner"], s["t"] = r, 16
    r.policy.set_precision(case.get("precision", "bf16"))
    for t in range(16):  # the cars have left their spawn points
        r.step(False, t)
    s["out"] = _sim_views(r.sim)
    if kind == "rollout":
        if case["chains"]:
            r.sim.set_chains(case["chains"])
        else:
            r.sim.set_fused_rollout(True)
        r.rollout_kernel_count(case["steps"])  # the graph is captured once, as a program's first rollout does
    elif kind in ("ppo_rollout", "ppo_update"):
        tr = s["trainer"] = W.Trainer(case["cars"], beams=case["beams"], rollout=case["rollout"])
        if kind == "ppo_rollout":
            s["out"] = {name: _view(getattr(tr, name)) for name in ("obs", "actions", "logp", "value", "reward", "done",
                                                                     "advantage")}
            s["out"]["state"] = _view(r.sim.state)
        else:
            tr.rollout(r.sim, r.policy, r.acts, 0)
            for _ in range(2):  # a program's later updates replay what its second one captured
                tr.update(r.policy)
            s["out"] = {"theta": _view(r.policy.theta), "grad": _view(tr.grad), "first": _view(tr.first),
                        "second": _view(tr.second)}
    elif kind == "learned_rollout":
        sur = s["sur"] = W.Surrogate(r.sim, hidden=512, batch=1024, seed=1, frame=case["frame"])
        sur.theta.write(_learned_theta(sur, _track(case["track"]), seed))
        sur.set_poses(1024, seed=seed)
        sur.train(1, lr=1e-30)  # takes the weights over
        r.rollout_surrogate(sur, case["steps"], step0=0)
    r.synchronize()
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "track":
        if "image" in s:
            free, loop, x0, y0, ramps = s["image"]
            return track_compile.compile_image(free, loop, x0, y0, case["cell"], ramps)
        route, half_width, bank, ramps = s["route"]
        return track_compile.ribbon(route, half_width, bank, case["cell"], ramps)
    out = s["out"]
    if kind == "policy":
        s["policy"].forward(s["x"], s["acts"])
        s["policy"].backward(s["x"], s["acts"], s["d3"], *s["back"])
        return out
    if kind == "learned_gradient":
        return dict(out, mse=s["sur"].gradient(0, s["labels"]))
    r, t = s["runner"], s["t"]
    if kind in ("step", "batch"):
        r.step(False, t)
        s["t"] = t + 1
        return out
    if kind == "ppo_update":
        return dict(out, kl=s["trainer"].update(r.policy))
    if kind == "ppo_rollout":
        reward = s["trainer"].rollout(r.sim, r.policy, r.acts, t)
        s["t"] = t + 1
        return dict(out, mean_reward=reward)
    if kind == "rollout":
        r.rollout(case["steps"], False, t)
    else:
        r.rollout_surrogate(s["sur"], case["steps"], step0=t)
    s["t"] = t + case["steps"]
    return out


def _step_work(track, cars, beams, forward=True):
    """One Runner step: the state, actions and observations read and written, the policy's weights and products, the
    physics and the beams' probes (the track's cells, a few MB, are read from cache)."""
    n = beams + 5
    beam = BEAM_FLOPS + PROBE_FLOPS * PROBES[track]
    flops = cars * (beams * beam + CAR_FLOPS)
    bytes_ = 4 * cars * (2 * 11 + 2 + 2 + n)
    if forward:
        flops += 2 * cars * (H * n + H * HA + OUT * HA)
        bytes_ += 4 * (cars * (n + OUT + 2) + H * n + H * HA + OUT * HA)
    return bytes_, flops


def work(case):
    kind = case["kind"]
    if kind == "track":
        cells = {"eight": 20.0 * 11.0, "oval": 16.0 * 16.0, "image": 24.0 * 24.0}[case["shape"]] / case["cell"] ** 2
        layers = 2 if case["shape"] == "eight" else 1
        return {"bytes": cells * (12.0 * layers + (case["shape"] == "image")), "flops": cells * layers * 120.0}
    if kind == "policy":
        n, cols = case["beams"] + 5, case["cols"]
        weights = H * n + H * HA + OUT * HA
        return {"bytes": 4.0 * (cols * (n + 4 * HA + 2 * OUT) + 2 * weights),
                "flops": 2.0 * cols * (2 * weights + H * HA + OUT * HA)}
    if kind == "batch":
        parts = [_step_work(t, c, case["beams"]) for t, c in zip(BATCH_TRACKS, _batch_cars(case["cars"]))]
        return {"bytes": float(sum(p[0] for p in parts)), "flops": float(sum(p[1] for p in parts))}
    if kind == "learned_gradient":
        nout = 4 * (case["beams"] - 1) // 3 if case["frame"] == "world" else case["beams"]
        h, b = case["hidden"], case["batch"]
        weights = h * 64 + 2 * h * h + nout * h
        return {"bytes": 4.0 * (2 * weights + b * (8 + case["beams"])), "flops": 6.0 * b * weights}
    cars, beams = case["cars"], case["beams"]
    if kind == "step":
        b, f = _step_work(case["track"], cars, beams)
    elif kind == "rollout":
        b, f = (case["steps"] * v for v in _step_work(case["track"], cars, beams))
    elif kind == "ppo_rollout":
        b, f = (case["rollout"] * v for v in _step_work(case["track"], cars, beams))
    elif kind == "ppo_update":
        n, samples = beams + 5, cars * case["rollout"]
        weights = H * n + H * HA + OUT * HA
        # four epochs over the storage: the inputs once as 32-bit observations, then as 16-bit operands in each
        b = samples * (4 * n + 4 * (2 * n + 4 * 6)) + 16 * 4 * 8 * weights
        f = 4 * 2 * samples * (2 * weights + H * HA + OUT * HA)
    else:
        nout = 4 * (beams - 1) // 3 if case["frame"] == "world" else beams
        audits = (case["steps"] + 15) // 16
        exact = _step_work(case["track"], cars, beams)
        plain = _step_work(case["track"], cars, 0)
        b = case["steps"] * exact[0]
        f = case["steps"] * (plain[1] + 2 * cars * (H * beams + 512 * 64 + 2 * 512 * 512 + 512 * nout))
        f += audits * (exact[1] - plain[1])
    return {"bytes": float(b), "flops": float(f)}


def exact(case, seed):
    if case["kind"] != "policy":
        return None
    theta, x, d3 = (torch.from_numpy(v).cuda().double() for v in _policy_inputs(case, seed))
    n, cols = case["beams"] + 5, case["cols"]
    w0, w1, w2, _ = torch.split(theta, [H * n, H * HA, OUT * HA, 2])
    w0, w1, w2 = w0.view(H, n), w1.view(H, HA), w2.view(OUT, HA)
    one = torch.ones((1, cols), dtype=torch.float64, device="cuda")
    h1 = torch.cat([torch.tanh(w0 @ x), one])
    h2 = torch.cat([torch.tanh(w1 @ h1), one])
    d2 = (w2.T @ d3) * (1 - h2 * h2)
    d1 = (w1.T @ d2[:H]) * (1 - h1 * h1)
    grad = torch.cat([(d1[:H] @ x.T).ravel(), (d2[:H] @ h1.T).ravel(), (d3 @ h2.T).ravel(),
                      torch.zeros(2, dtype=torch.float64, device="cuda")])
    return {"h1": h1, "h2": h2, "o": w2 @ h2, "d2": d2, "d1": d1, "grad": grad}
