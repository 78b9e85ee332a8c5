"""The direct broadphase (a warp per owner over its world's bodies) on both sides of its line and at the
edges of its warps, tiles, kept partners and body order: pair keys, manifolds and state equal the
oracle's, whose pairs come from the reference's tree (collision/broadphase/DbvtBroadphase.java:89-150,
HashedOverlappingPairCache.java:179-188)."""
import numpy as np
import pytest

import harness as H
import pyoracle
from jbgpu import _abi, scenes

pytestmark = pytest.mark.gpu


def _step_both(gpu_lib, sc, steps):
    g = gpu_lib.GpuWorld(sc)
    o = pyoracle.OracleWorld(sc)
    for st in range(steps):
        for stage in (_abi.STAGE_APPLY_GRAVITY, _abi.STAGE_PREDICT, _abi.STAGE_AABB, _abi.STAGE_PAIRS,
                      _abi.STAGE_NARROWPHASE):
            g.stage(stage, sc.dt)
            o.stage(stage, sc.dt)
        assert not H.compare_manifolds(o.get_manifolds(), g.get_manifolds()), st
        for stage in (_abi.STAGE_ISLANDS, _abi.STAGE_SOLVE, _abi.STAGE_INTEGRATE, _abi.STAGE_ACTIVATION):
            o.stage(stage, sc.dt)   # the oracle's: a body here has more contacts than the GPU solver has colours
        H.copy_world(o, g)
    pairs = g.counters()["pairs"]
    g.close()
    return pairs


def _spheres(n, worlds, big, seed):
    """n spheres over `worlds` batch worlds in shuffled order, static planes before and between them,
    filter groups, and `big` spheres a world that overlap every body of it."""
    rng = np.random.Generator(np.random.PCG64(seed))
    shapes = [dict(scenes.PLANE), {"type": _abi.SHAPE_SPHERE, "params": (0.5, 0.0, 0.0, 0.0), "points": None},
              {"type": _abi.SHAPE_SPHERE, "params": (90.0, 0.0, 0.0, 0.0), "points": None}]
    b = scenes._bodies(n)
    b["shape"] = 1
    b["mass"] = 1.0
    b["local_inertia"] = 0.1
    b["world"] = rng.integers(0, worlds, n)
    side = max(2, int(round((n / worlds) ** (1.0 / 3.0))))
    scenes._set_transforms(b, scenes.random_rotations(rng, n), rng.uniform(0.0, 0.8 * side, (n, 3)))
    b["collision_group"][::7] = 64
    b["collision_mask"][::7] = 1 | 2
    for wi in range(worlds):
        mine = np.nonzero(b["world"] == wi)[0]
        b["shape"][mine[:big]] = 2
        b["transform"][mine[:big], 9:] = (0.0, 95.0, 0.0)
    planes = np.concatenate([scenes._plane_body(0) for _ in range(worlds)])
    planes["world"] = np.arange(worlds)
    cut = n // 2
    bodies = np.concatenate([planes[: worlds // 2], b[:cut], planes[worlds // 2:], b[cut:]])
    return scenes.Scene("direct", 1.0 / 60.0, 1, {"gravity": (0.0, -9.81, 0.0), "num_iterations": 2}, shapes, bodies)


@pytest.mark.parametrize("n,worlds,big", [(1, 1, 0), (2, 1, 0), (31, 1, 1), (33, 1, 0), (255, 1, 1), (257, 1, 2), (300, 1, 1),
                                          (1023, 1, 1), (1025, 1, 0), (2049, 1, 0), (4095, 1, 0), (4096, 1, 0),
                                          (7800, 1, 0), (8100, 1, 0), (700, 9, 1), (900, 300, 0), (40000, 4000, 0)])
def test_pairs_same_as_the_oracle(gpu_lib, oracle_lib, n, worlds, big):
    assert _step_both(gpu_lib, _spheres(n, worlds, big, n + worlds), 2) >= 0


@pytest.mark.parametrize("n,compounds", [(30, 12), (400, 40)])
def test_compounds_and_meshes(gpu_lib, oracle_lib, n, compounds):
    assert _step_both(gpu_lib, scenes.terrain(n, compounds=compounds, seed=n), 6) > 0


def test_queries_between_steps(gpu_lib, oracle_lib):
    """Rays and steps by turns: the queries build the tree of the current order when they need it."""
    sc = scenes.small_mixed(n=120, seed=11)
    g = gpu_lib.GpuWorld(sc)
    h = gpu_lib.GpuWorld(sc)
    rng = np.random.Generator(np.random.PCG64(3))
    frm = rng.uniform((-5, 0, -5), (5, 10, 5), (9000, 3)).astype(np.float32)
    to = rng.uniform((-5, -1, -5), (5, 10, 5), (9000, 3)).astype(np.float32)
    for k in range(14):
        g.step(sc.dt)
        h.step(sc.dt)
        if k % 3 == 2:
            o = pyoracle.OracleWorld(sc)
            H.copy_world(g, o, manifolds=False)
            a, b = o.ray_test(frm, to), g.ray_test(frm, to)
            assert np.array_equal(a.view(np.uint8), b.view(np.uint8)), k
    assert not H.compare_state(g.get_state(), h.get_state())
    g.close()
    h.close()
