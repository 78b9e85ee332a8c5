"""Ray batches on both sides of the line between a block per ray and the candidate lists, (bodies + 1,600) x rays
at 7.2 million: 2,880 rays among 900 bodies are the last by blocks, 7,200,000 / 1,601 among one."""
import numpy as np
import pytest

import pyoracle
from test_ray_paths import F, REACH, _row_of_spheres, _same
from jbgpu.lib import GpuWorld

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bodies,n", [(900, 2880), (900, 2881), (1, 4497), (1, 4498)])
def test_both_sides(gpu_lib, oracle_lib, bodies, n):
    sc = _row_of_spheres(bodies, 4)
    rng = np.random.Generator(np.random.PCG64(n))
    frm = np.stack([rng.uniform(-2, 2 + 0.05 * bodies, n), np.full(n, 6.0), rng.uniform(-1.2, 1.2, n)], 1).astype(F)
    to = frm.copy()
    to[:, 1] = -6.0
    for i, reach in enumerate(REACH):
        frm[i] = (-5.0, 0.3, 0.1)
        to[i] = (-1.06 + 0.05 * reach, 0.3, 0.1)
    g = GpuWorld(sc)
    want = pyoracle.OracleWorld(sc).ray_test(frm, to)
    assert np.any(want["body"] >= 0)
    assert _same(want, g.ray_test(frm, to))
    g.close()
