"""Ray batches on both sides of the line between the two ray paths (a block per ray over all bodies;
the tree walk with candidate lists and rounds of casts): the hit records are the oracle's bit for
bit (CollisionWorld.rayTest with a ClosestRayResultCallback, collision/dispatch/
CollisionWorld.java:553-591)."""
import numpy as np
import pytest

from jbgpu import _abi, scenes
from jbgpu.lib import GpuWorld

import harness as H
import pyoracle

F = np.float32


def _same(a, b):
    return np.array_equal(a.view(np.uint8).reshape(len(a), -1), b.view(np.uint8).reshape(len(b), -1))


def _row_of_spheres(k, seed):
    """k overlapping static spheres along x in shuffled body order, some at the same place."""
    rng = np.random.Generator(np.random.PCG64(seed))
    shapes = [{"type": _abi.SHAPE_SPHERE, "params": (1.0, 0.0, 0.0, 0.0), "points": None}]
    b = np.concatenate([scenes._bodies(1) for _ in range(k)])
    b["shape"] = 0
    x = rng.permutation(np.arange(k) // 2 * 2) * 0.05
    b["transform"][:, 9:] = np.stack([x, 2e-6 * rng.integers(0, 5, k), np.zeros(k)], 1)
    return scenes.Scene("row", 1.0 / 60.0, 1, {}, shapes, b)


# candidates of a ray at the edges of the per-ray lists (256), the entry sort (128), a warp (32) and the block's list (768)
REACH = (0, 1, 2, 31, 32, 33, 127, 128, 129, 255, 256, 257, 767, 768, 769, 900)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 33, 600, 6122, 6123, 9000])   # (900 + 4000) x 6122 is the last batch by blocks
def test_ray_paths_long_lists(gpu_lib, oracle_lib, n):
    sc = _row_of_spheres(900, 4)
    rng = np.random.Generator(np.random.PCG64(5))
    frm = np.stack([rng.uniform(-2, 47, n), np.full(n, 6.0), rng.uniform(-1.2, 1.2, n)], 1).astype(F)
    to = frm.copy()
    to[:, 1] = -6.0
    for i, reach in enumerate(REACH[:n]):                # along the row, ending at its reach-th sphere
        frm[i] = (-5.0, 0.3, 0.1)
        to[i] = (-1.06 + 0.05 * reach, 0.3, 0.1)
    g = GpuWorld(sc)
    assert _same(pyoracle.OracleWorld(sc).ray_test(frm, to), g.ray_test(frm, to))
    g.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [7, 12001])
def test_ray_paths_meshes_compounds_and_filters(gpu_lib, oracle_lib, n):
    sc = scenes.terrain(40, compounds=16, seed=6)
    g = GpuWorld(sc)
    for _ in range(40):
        g.step(sc.dt)
    o = pyoracle.OracleWorld(sc)
    H.copy_world(g, o, manifolds=False)
    rng = np.random.Generator(np.random.PCG64(8))
    frm = rng.uniform(-8, 8, (n, 3)).astype(F)
    to = rng.uniform(-8, 8, (n, 3)).astype(F)
    to[: n // 2] = frm[: n // 2]
    to[: n // 2, 1] = -9.0
    to[-1] = frm[-1]                                     # a ray of no length
    assert _same(o.ray_test(frm, to), g.ray_test(frm, to))
    assert _same(o.ray_test(frm, to, group=1, mask=2), g.ray_test(frm, to, group=1, mask=2))
    g.close()


@pytest.mark.gpu
@pytest.mark.parametrize("n", [9, 12001])
def test_ray_paths_batched_worlds(gpu_lib, oracle_lib, n):
    sc = scenes.hinged_chains(chains=3, links=4, loose=6, seed=6, worlds=4)
    g = GpuWorld(sc)
    for _ in range(20):
        g.step(sc.dt)
    o = pyoracle.OracleWorld(sc)
    H.copy_world(g, o, manifolds=False)
    rng = np.random.Generator(np.random.PCG64(9))
    frm = rng.uniform((-4, 0, -4), (4, 12, 4), (n, 3)).astype(F)
    to = rng.uniform((-4, -1, -4), (4, 12, 4), (n, 3)).astype(F)
    world = rng.integers(0, 4, n).astype(np.int32)
    assert _same(o.ray_test(frm, to, world=world), g.ray_test(frm, to, world=world))
    g.close()


@pytest.mark.gpu
def test_rays_before_the_first_step_leave_the_same_order(gpu_lib):
    """A query on bodies added since the last step fixes the order the solver's parts follow, whichever
    path the rays take: a world of several parts steps the same after few rays and after many."""
    sc = scenes.small_mixed(2600, seed=3, region=(14.0, 16.0, 14.0))
    rng = np.random.Generator(np.random.PCG64(2))
    worlds = [GpuWorld(sc), GpuWorld(sc)]
    for g, n in zip(worlds, (3, 12000)):
        frm = rng.uniform((-7, 0, -7), (7, 16, 7), (n, 3)).astype(F)
        to = rng.uniform((-7, 0, -7), (7, 16, 7), (n, 3)).astype(F)
        g.ray_test(frm, to)
        for _ in range(40):
            g.step(sc.dt)
    assert worlds[0].counters()["cut_manifolds"] > 0
    assert not H.compare_state(worlds[0].get_state(), worlds[1].get_state())
    for g in worlds:
        g.close()
