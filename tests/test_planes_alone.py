"""Worlds of static planes alone have no tree; batches of rays on both paths find the planes."""
import numpy as np
import pytest

import pyoracle
from jbgpu import scenes

pytestmark = pytest.mark.gpu
F = np.float32


@pytest.mark.parametrize("n", [5, 9000])
def test_rays_on_planes(gpu_lib, oracle_lib, n):
    sc = scenes.Scene("planes", 1.0 / 60.0, 1, {"gravity": (0.0, -9.81, 0.0)}, [dict(scenes.PLANE)],
                      np.concatenate([scenes._plane_body(0)] * 2))
    g, o = gpu_lib.GpuWorld(sc), pyoracle.OracleWorld(sc)
    rng = np.random.Generator(np.random.PCG64(n))
    frm = rng.uniform(-5, 5, (n, 3)).astype(F)
    to = rng.uniform(-5, 5, (n, 3)).astype(F)
    want = o.ray_test(frm, to)
    assert np.any(want["body"] >= 0)
    for _ in range(2):
        assert np.array_equal(want.view(np.uint8), g.ray_test(frm, to).view(np.uint8))
        g.step(sc.dt)
    g.close()
