"""Workloads of the rigid-body library that its speed is judged on, through the calls a program makes.

A program keeps a GpuWorld over its simulation, steps it once per frame (stepSimulation) and reads the
bodies' transforms back for drawing, or the whole state for a controller; it casts rays and sweeps
at the world, and it trains the warm-start network on contact samples.  The world cases start from
a pile that has come to rest against its ground and keep simulating it (deactivation off, as a
program sets it whose bodies have to stay responsive), so that one pass costs what the next one does.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "libgdx-jbullet_gb300"))

from jbgpu import _abi, scenes  # noqa: E402
from jbgpu.lib import MLP_INPUTS, MLP_OUTPUTS, MLP_PARAMS, GpuWorld, Mlp  # noqa: E402


def listed():
    return [
        # a room of a few dozen bodies of every convex kind: a frame is launches and latency
        {"name": "room_60", "kind": "step", "scene": "small", "bodies": 60, "substeps": 1},
        # the 1,000-box pile of the benchmark, two substeps a frame as stacking scenes use
        {"name": "boxes_1000", "kind": "step", "scene": "boxes", "bodies": 1000, "substeps": 2},
        # ropes and ragdolls: 64 chains of 8 links on ball joints, with loose boxes among them
        {"name": "chains_64x8", "kind": "step", "scene": "ball", "bodies": 64, "links": 8, "substeps": 1},
        # a large game level of spheres, boxes and capsules (odd count)
        {"name": "mixed_20001", "kind": "step", "scene": "mixed", "bodies": 20001, "substeps": 1},
        # the benchmark's headline size
        {"name": "mixed_100000", "kind": "step", "scene": "mixed", "bodies": 100000, "substeps": 1},
        # rubble: convex hulls of 32 points, the narrowphase's hardest pairs
        {"name": "hulls_4000", "kind": "step", "scene": "hulls", "bodies": 4000, "substeps": 1},
        # convex and compound bodies on a triangle-mesh landscape
        {"name": "terrain_4000", "kind": "step", "scene": "terrain", "bodies": 4000, "compounds": 400, "substeps": 1},
        # a quarter of the benchmark's 4,096 independent worlds of 16 to 2,048 bodies
        {"name": "worlds_1024", "kind": "step", "scene": "worlds", "bodies": 2048, "worlds": 1024, "substeps": 1},
        # a controller over 256 small worlds: forces in, two substeps, the whole state out
        {"name": "control_256", "kind": "control", "scene": "worlds", "bodies": 128, "worlds": 256, "substeps": 2},
        # line of sight and picking: a few rays a frame from host memory
        {"name": "rays_host_64", "kind": "rays", "scene": "mixed", "bodies": 2000, "count": 64, "device": False},
        # a sensor's rays against a large level, on device buffers
        {"name": "rays_device_200k", "kind": "rays", "scene": "mixed", "bodies": 20000, "count": 200000, "device": True},
        # one mini-batch of the warm-start network's training: forward and backward
        {"name": "network_16384", "kind": "network", "count": 16384},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["small", "boxes", "mixed", "mixed", "hulls", "terrain", "worlds", "joints", "control", "rays", "rays",
                       "network"])
    if what == "small":
        return {"kind": "step", "scene": "small", "bodies": _log(rng, 24, 400), "substeps": rng.choice([1, 2])}
    if what == "boxes":
        return {"kind": "step", "scene": "boxes", "bodies": _log(rng, 100, 4000), "substeps": rng.choice([1, 2])}
    if what == "mixed":
        return {"kind": "step", "scene": "mixed", "bodies": _log(rng, 500, 90000), "substeps": 1}
    if what == "hulls":
        return {"kind": "step", "scene": "hulls", "bodies": _log(rng, 200, 4000), "substeps": 1}
    if what == "terrain":
        n = _log(rng, 200, 4000)
        return {"kind": "step", "scene": "terrain", "bodies": n, "compounds": rng.randrange(0, n // 8 + 1), "substeps": 1}
    if what == "worlds":
        return {"kind": "step", "scene": "worlds", "bodies": _log(rng, 64, 1500), "worlds": _log(rng, 32, 1000), "substeps": 1}
    if what == "joints":
        return {"kind": "step", "scene": rng.choice(["ball", "hinge", "sixdof", "cone"]), "bodies": _log(rng, 4, 100),
                "links": rng.randrange(3, 10), "substeps": rng.choice([1, 2])}
    if what == "control":
        return {"kind": "control", "scene": "worlds", "bodies": _log(rng, 32, 256), "worlds": _log(rng, 16, 400),
                "substeps": rng.choice([1, 2, 4])}
    if what == "rays":
        n = _log(rng, 1, 200000)
        return {"kind": "rays", "scene": "mixed", "bodies": _log(rng, 500, 20000), "count": n, "device": rng.random() < 0.5}
    return {"kind": "network", "count": _log(rng, 64, 65536)}


def _layers(n, side, pitch, y0, rng):
    """Places for n bodies, dropped layer by layer on a square of the given side: no two of them touch."""
    row = max(1, round(side / pitch))
    cell = np.arange(n)
    ij = np.stack([cell % row, cell // row % row], 1) * pitch - 0.5 * (row - 1) * pitch
    pos = np.stack([ij[:, 0], y0 + (cell // (row * row)) * pitch, ij[:, 1]], 1)
    return (pos + rng.uniform(-0.02, 0.02, (n, 3)))[rng.permutation(n)]


def _drop(scene, side, pitch, seed):
    """The scene's movable bodies laid out in layers over each world's ground, turned at random."""
    rng = np.random.Generator(np.random.PCG64(seed + 1))
    b = scene.bodies
    starts = np.flatnonzero(np.r_[True, b["world"][1:] != b["world"][:-1]])
    for first, end in zip(starts, np.r_[starts[1:], len(b)]):
        b["transform"][first + 1:end, 9:] = _layers(end - first - 1, side, pitch, 1.2, rng)
    moving = b["mass"] > 0
    b["transform"][moving, :9] = scenes.random_rotations(rng, int(moving.sum())).reshape(-1, 9)
    return scene


def _scene(case, seed):
    """The scene of a case and the steps after which it lies on its ground."""
    n, what = case["bodies"], case["scene"]
    if what == "small":
        side = 6.0 * math.sqrt(n / 60.0)
        return _drop(scenes.small_mixed(n, seed=seed), max(side, 6.0), 2.2, seed), 150
    if what == "boxes":
        side = 20.0 * math.sqrt(n / 1000.0)
        return _drop(scenes.boxes_on_plane(n, seed=seed), max(side, 4.0), 1.8, seed), 180
    if what == "mixed":
        side = 200.0 * math.sqrt(n / 100000.0)
        return _drop(scenes.mixed_100k(n, seed=seed), max(side, 6.0), 2.2, seed), 360
    if what == "hulls":
        return scenes.hulls(n, seed=seed, box=max(12.0, 2.2 * n ** (1.0 / 3.0))), 210
    if what == "terrain":
        side = 90.0 * math.sqrt(n / 4000.0)
        return scenes.terrain(n, seed=seed, cells=max(8, int(side * 0.7)), size=side * 1.15, compounds=case["compounds"],
                              region=(side, 15.0, side), y0=4.0, bowl=0.05), 150
    if what == "worlds":   # the worlds' sizes belong to the case, where their bodies start to the seed
        side = 20.0 * math.sqrt(n / 2048.0)
        return _drop(scenes.batched_worlds(case["worlds"], seed=0, nmin=16, nmax=n), max(side, 3.6), 1.8, seed), 200
    make = {"ball": scenes.jointed_chains, "hinge": scenes.hinged_chains, "sixdof": scenes.sixdof_chains,
            "cone": scenes.cone_chains}[what]
    return make(n, case["links"], loose=2 * n, seed=seed), 60


def _world(case, seed):
    scene, settle = _scene(case, seed)
    world = GpuWorld(scene, config=_abi.default_config(disable_deactivation=1, **scene.config))
    for _ in range(settle):
        world.step(scene.dt)
    return world, scene


def _rays(world, count, seed):
    """Half of the rays straight down from above the bodies, half between random points among them."""
    pos = world.get_transforms()[1:, 9:]
    pos = pos[np.all(np.abs(pos) < 1e6, axis=1)]
    lo, hi = np.percentile(pos, 1, axis=0), np.percentile(pos, 99, axis=0)
    hi[1] = max(hi[1], lo[1] + 1.0)
    rng = np.random.default_rng(seed)
    a, b = (rng.uniform(lo, hi, (count, 3)).astype(np.float32) for _ in range(2))
    down = (count + 1) // 2
    a[:down, 1] = hi[1] + 5.0
    b[:down] = a[:down]
    b[:down, 1] = lo[1] - 2.0
    return a, b


def _network_inputs(case, seed):
    """Weights as a training run starts from, and contact samples spread like the features' scales."""
    rng = np.random.default_rng(seed)
    h = 64
    layers = [(h, MLP_INPUTS), (h, h), (MLP_OUTPUTS, h)]
    parts = []
    for out, inp in layers:
        a = math.sqrt(6.0 / (out + inp))
        parts += [rng.uniform(-a, a, out * inp), rng.uniform(-0.05, 0.05, out)]
    params = np.concatenate(parts).astype(np.float32)
    norm = np.concatenate([rng.normal(0.0, 0.1, MLP_INPUTS), rng.uniform(0.5, 2.0, MLP_INPUTS),
                           rng.normal(0.0, 0.1, MLP_OUTPUTS), rng.uniform(0.5, 2.0, MLP_OUTPUTS), [1.0]]).astype(np.float32)
    x = (rng.standard_normal((case["count"], MLP_INPUTS)) * 2.0).astype(np.float32)
    t = rng.standard_normal((case["count"], MLP_OUTPUTS)).astype(np.float32)
    return params, norm, x, t


def prepare(case, seed):
    if case["kind"] == "network":
        params, norm, x, t = _network_inputs(case, seed)
        net = Mlp(seed=seed)
        net.set_params(params, norm)
        return {"case": case, "net": net, "x": x, "t": t}
    world, scene = _world(case, seed)
    state = {"case": case, "world": world, "dt": scene.dt}
    n = world.n_bodies
    if case["kind"] != "rays":   # stepSimulation's clock starts a frame ahead: let it run level
        for _ in range(2):
            world.step_simulation(case["substeps"] * scene.dt, case["substeps"], scene.dt)
    if case["kind"] == "step":
        state["out"] = torch.empty((n, 12), pin_memory=True).numpy()
    elif case["kind"] == "control":
        force = torch.empty((n, 3), pin_memory=True).numpy()
        force[...] = np.random.default_rng(seed).uniform(-2.0, 2.0, (n, 3))
        state["force"] = force
    else:
        a, b = _rays(world, case["count"], seed)
        if case["device"]:
            state["from"], state["to"] = torch.from_numpy(a).cuda(), torch.from_numpy(b).cuda()
            state["hits"] = torch.empty((case["count"], 8), device="cuda")
        else:
            state["from"], state["to"] = a, b
    return state


def run(state):
    case = state["case"]
    if case["kind"] == "network":
        grad, loss = state["net"].gradients(state["x"], state["t"])
        return {"grad": grad, "loss": loss}
    world, k, dt = state["world"], case.get("substeps"), state["dt"]
    if case["kind"] == "step":
        world.step_simulation(k * dt, k, dt)
        return {"transforms": world.get_transforms(state["out"])}
    if case["kind"] == "control":
        world.apply_forces(state["force"])
        world.step_simulation(k * dt, k, dt)
        return world.get_state()
    if case["device"]:
        h = state["hits"]
        world.ray_test_device(state["from"].data_ptr(), state["to"].data_ptr(), case["count"], h.data_ptr())
        return {"body": h.view(torch.int32)[:, 0], "hit": h[:, 1:]}
    h = world.ray_test(state["from"], state["to"])
    return {k: h[k] for k in ("body", "fraction", "normal", "point")}


# Overlapping pairs and contact points per body of the settled scenes, rounded (for work()).
_PAIRS = {"small": 4.0, "boxes": 6.0, "mixed": 5.0, "hulls": 9.0, "terrain": 4.0, "worlds": 4.0, "ball": 1.5, "hinge": 1.5,
          "sixdof": 1.5, "cone": 1.5}
_POINTS = {"small": 3.0, "boxes": 4.0, "mixed": 2.5, "hulls": 4.0, "terrain": 2.0, "worlds": 3.0, "ball": 1.0, "hinge": 1.0,
           "sixdof": 1.0, "cone": 1.0}


def work(case):
    if case["kind"] == "network":
        n = case["count"]
        return {"bytes": 4 * n * (MLP_INPUTS + MLP_OUTPUTS) + 8 * MLP_PARAMS, "flops": 3 * 2 * n * (64 * 24 + 64 * 64 + 3 * 64)}
    if case["kind"] == "rays":
        n, b = case["count"], case["bodies"]
        # rays in, hits out, each body's box and transform once; a walk of about 2 log2(b) boxes a ray
        return {"bytes": 56 * n + 80 * b, "flops": n * 24 * 2 * math.log2(b + 2)}
    what = case["scene"]
    if what == "worlds":   # sizes are spread evenly over their logarithm from 16 to `bodies`
        n = case["worlds"] * (case["bodies"] - 16) / math.log(case["bodies"] / 16.0)
    elif what in ("ball", "hinge", "sixdof", "cone"):
        n = case["bodies"] * (case["links"] + 2)
    else:
        n = case["bodies"] + case.get("compounds", 0)
    pairs, points, k = _PAIRS[what] * n, _POINTS[what] * n, case["substeps"]
    iters = 15 if what == "hulls" else 10
    # per substep: a body's state read and written once, a pair's key and a contact point's record
    # read and written once; three solver rows per point and iteration of about 60 operations
    nbytes = k * (400 * n + 16 * pairs + 256 * points) + (168 if case["kind"] == "control" else 48) * n
    return {"bytes": nbytes, "flops": k * (600 * n + 300 * pairs + points * 3 * 60 * (iters + 1))}


def exact(case, seed):
    """The network's gradient and loss in 64 bits.  A step of a world and a cast ray have no such value
    apart from the simulation that leads to them."""
    if case["kind"] != "network":
        return None
    params, norm, x, t = (a.astype(np.float64) for a in _network_inputs(case, seed))
    at, w = 0, []
    for out, inp in ((64, MLP_INPUTS), (64, 64), (MLP_OUTPUTS, 64)):
        w.append((params[at:at + out * inp].reshape(out, inp), params[at + out * inp:at + out * (inp + 1)]))
        at += out * (inp + 1)
    (w1, b1), (w2, b2), (w3, b3) = ((torch.from_numpy(m).requires_grad_(), torch.from_numpy(b).requires_grad_()) for m, b in w)
    i, o = MLP_INPUTS, MLP_OUTPUTS
    xin = torch.from_numpy(np.arcsinh((x - norm[:i]) * norm[i:2 * i]))
    target = torch.from_numpy((t - norm[2 * i:2 * i + o]) / norm[2 * i + o:2 * i + 2 * o])
    gelu = torch.nn.GELU(approximate="tanh")
    y = gelu(gelu(xin @ w1.T + b1) @ w2.T + b2) @ w3.T + b3
    loss = ((y - target) ** 2).mean()
    loss.backward()
    return {"grad": torch.cat([p.grad.reshape(-1) for p in (w1, b1, w2, b2, w3, b3)]), "loss": float(loss.detach())}
