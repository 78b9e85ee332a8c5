"""Ray batches by lists whose candidates are cast at once (up to six a ray on average, two with triangle meshes)
and in rounds, on both sides of the line: hit records equal the oracle's.  Overlapping spheres in a row put
every ray through as many boxes as wanted; on a landscape its box is one candidate more."""
import numpy as np
import pytest

import pyoracle
from jbgpu import _abi, scenes
from jbgpu.lib import GpuWorld

pytestmark = pytest.mark.gpu
F = np.float32


def _clusters(deep, mesh):
    """Stacks of `deep` overlapping spheres; rays run down through them."""
    shapes = [{"type": _abi.SHAPE_SPHERE, "params": (0.5, 0.0, 0.0, 0.0), "points": None}]
    b = scenes._bodies(40 * deep)
    k = np.arange(40 * deep)
    b["transform"][:, 9:] = np.stack([3.0 * (k // deep % 8), 0.3 * (k % deep) + 3.0, 3.0 * (k // (8 * deep))], 1)
    b = b[np.random.Generator(np.random.PCG64(deep)).permutation(len(b))]
    if mesh:
        land = scenes.terrain(1, seed=3, size=60.0)
        ground = next(s for s in land.shapes if s["type"] == _abi.SHAPE_TRIANGLE_MESH)
        shapes.append(ground)
        g = scenes._bodies(1)
        g["shape"] = 1
        b = np.concatenate([b, g])
    return scenes.Scene("clusters", 1.0 / 60.0, 1, {}, shapes, b)


@pytest.mark.parametrize("mesh", [False, True])
@pytest.mark.parametrize("deep", [1, 2, 5, 6, 7, 40])
def test_at_once_and_in_rounds(gpu_lib, oracle_lib, deep, mesh):
    sc, n = _clusters(deep, mesh), 9000
    rng = np.random.Generator(np.random.PCG64(7))
    which = rng.integers(0, 40, n)
    frm = np.stack([3.0 * (which % 8) + rng.uniform(-0.4, 0.4, n), np.full(n, 30.0),
                    3.0 * (which // 8) + rng.uniform(-0.4, 0.4, n)], 1).astype(F)
    to = frm.copy()
    to[:, 1] = -30.0
    up = rng.random(n) < 0.3                      # some from below, some across
    frm[up], to[up] = to[up].copy(), frm[up].copy()
    to[::11] += F(4.0)
    g = GpuWorld(sc)
    want = pyoracle.OracleWorld(sc).ray_test(frm, to)
    assert np.mean(want["body"] >= 0) > 0.5
    assert np.array_equal(want.view(np.uint8), g.ray_test(frm, to).view(np.uint8))
    g.close()
