"""Rays cast on bodies that changed since the last step, in worlds large enough for the tree's pairs (past
the direct broadphase's line).  Few rays need the body order alone and leave the tree to the next step:
its pairs are those of a brute-force search, and state is the same as after many rays, whose path makes
the tree.  With and without step graphs, before the first step, after bodies were taken out and added, and
when the order is due for renewal.  Worlds of listed bodies alone have no tree; many rays find the planes."""
import numpy as np
import pytest

import harness as H
import pyoracle
from jbgpu import _abi, scenes

pytestmark = pytest.mark.gpu
F = np.float32
SHAPES = [dict(scenes.PLANE), {"type": _abi.SHAPE_SPHERE, "params": (0.4, 0.0, 0.0, 0.0), "points": None},
          {"type": _abi.SHAPE_BOX, "params": (0.3, 0.35, 0.3, 0.0), "points": None}]
CONFIG = {"gravity": (0.0, -9.81, 0.0), "num_iterations": 4}


def _bodies(n, y0, seed):
    rng = np.random.Generator(np.random.PCG64(seed))
    b = scenes._bodies(n)
    b["shape"] = 1 + np.arange(n) % 2
    b["mass"] = 1.0
    b["local_inertia"] = 0.08
    scenes._set_transforms(b, scenes.random_rotations(rng, n), rng.uniform((-14, y0, -14), (14, y0 + 16, 14), (n, 3)))
    return b


def _rays(g, n):
    rng = np.random.Generator(np.random.PCG64(n))
    g.ray_test(rng.uniform((-14, 0, -14), (14, 20, 14), (n, 3)).astype(F),
               rng.uniform((-14, 0, -14), (14, 20, 14), (n, 3)).astype(F))


@pytest.mark.parametrize("graphs", [0, 1])
def test_steps_after_rays(gpu_lib, oracle_lib, graphs):
    sc = scenes.Scene("tree", 1.0 / 60.0, 1, CONFIG, SHAPES, np.concatenate([scenes._plane_body(0), _bodies(8300, 0.6, 1)]))
    more = scenes.Scene("more", 1.0 / 60.0, 1, CONFIG, SHAPES, _bodies(40, 18.0, 2))
    cfg = _abi.default_config(**dict(CONFIG, step_graphs=graphs))
    few, many = gpu_lib.GpuWorld(sc, config=cfg), gpu_lib.GpuWorld(sc, config=cfg)
    o = pyoracle.OracleWorld(sc)
    o.set_brute_force_pairs(True)

    def steps(k):
        for _ in range(k):
            few.step(sc.dt)
            many.step(sc.dt)
            st = few.get_state()
            o.set_state({f: st[f] for f in H.STATE_COPY})
            o.stage(_abi.STAGE_PAIRS, sc.dt)
            assert np.array_equal(o.get_pairs(), few.get_pairs())

    for change in (None, "remove", "add"):
        for w in (few, many, o):
            if change == "remove":
                w.remove_bodies(np.arange(50, 90, dtype=np.int32))
            elif change == "add":
                w.add_scene(more)
        _rays(few, 3)
        _rays(many, 12000)
        steps(2)                             # one on the order as the query made it
        _rays(few, 3)
        steps(4)                             # past the renewal
        assert not H.compare_state(few.get_state(), many.get_state()), change
    for g in (few, many):
        g.close()
