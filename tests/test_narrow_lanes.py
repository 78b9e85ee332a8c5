"""GJK with 32, 4 and 1 lanes to a pair (the pass picks by the pair capacity): manifolds and state equal
the oracle's bit for bit.  Hulls of 1 to 33 points, so that the lanes' vertex scans have remainders and
lanes without a vertex, among boxes, spheres and capsules."""
import numpy as np
import pytest

import harness as H
import pyoracle
from jbgpu import _abi, scenes

pytestmark = pytest.mark.gpu


def _scene(n, seed):
    """n bodies of cycling kinds on a jittered grid a little closer than they are large."""
    rng = np.random.Generator(np.random.PCG64(seed))
    shapes = [dict(scenes.PLANE),
              {"type": _abi.SHAPE_BOX, "params": (0.5, 0.4, 0.6, 0.0), "points": None},
              {"type": _abi.SHAPE_SPHERE, "params": (0.5, 0.0, 0.0, 0.0), "points": None},
              {"type": _abi.SHAPE_CAPSULE, "params": (0.3, 0.6, 0.0, 0.0), "points": None}]
    for k in (1, 2, 3, 4, 7, 8, 9, 31, 32, 33):
        d = rng.standard_normal((k, 3))
        shapes.append({"type": _abi.SHAPE_CONVEX_HULL, "params": (0.0, 0.0, 0.0, 0.0),
                       "points": (0.5 * d / np.linalg.norm(d, axis=1, keepdims=True)).astype(np.float32)})
    b = scenes._bodies(n)
    b["shape"] = 1 + np.arange(n) % (len(shapes) - 1)
    b["mass"] = 1.0
    b["local_inertia"] = 0.2
    side = max(2, int(round(n ** (1.0 / 3.0))))
    i = np.arange(n)
    grid = np.stack([i % side, i // (side * side), (i // side) % side], 1) * 0.95
    pos = grid + rng.uniform(-0.05, 0.05, (n, 3)) + (0.0, 0.7, 0.0)
    scenes._set_transforms(b, scenes.random_rotations(rng, n), pos)
    return scenes.Scene("lanes_%d" % n, 1.0 / 60.0, 1, {"gravity": (0.0, -9.81, 0.0), "num_iterations": 4}, shapes,
                        np.concatenate([scenes._plane_body(0), b]))


@pytest.mark.parametrize("n", [3, 90, 400, 1500, 6000])
def test_same_as_the_oracle(gpu_lib, oracle_lib, n):
    sc = _scene(n, n)
    g = gpu_lib.GpuWorld(sc)
    o = pyoracle.OracleWorld(sc)
    for st in range(3):
        for stage in (_abi.STAGE_APPLY_GRAVITY, _abi.STAGE_PREDICT, _abi.STAGE_AABB, _abi.STAGE_PAIRS,
                      _abi.STAGE_NARROWPHASE):
            g.stage(stage, sc.dt)
            o.stage(stage, sc.dt)
        assert not H.compare_manifolds(o.get_manifolds(), g.get_manifolds()), st
        assert g.counters()["gjk_calls"] == o.counters()["gjk_calls"]
        for stage in (_abi.STAGE_ISLANDS, _abi.STAGE_SOLVE, _abi.STAGE_INTEGRATE, _abi.STAGE_ACTIVATION):
            g.stage(stage, sc.dt)
        H.copy_world(g, o)
    assert g.counters()["gjk_calls"] > 0 and g.counters()["contacts"] > 0
    g.close()
