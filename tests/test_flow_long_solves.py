"""Solves of many iterations in batches whose worlds are cut into more pieces than blocks are resident: the
first piece of a world waits for its second until another world's blocks are through, seconds after 60,000
iterations, and the wait's bound grows with them.  All worlds are the same and end the same, and equal the
colour-by-colour solver (solver_smem_bodies below the part)."""
import numpy as np
import pytest

import harness as H
from jbgpu import _abi, scenes

pytestmark = pytest.mark.gpu


def _rows(worlds, n):
    """A row of n touching boxes on a plane in every world: neighbours lie in different pieces."""
    b = scenes._bodies(n)
    b["shape"] = 1
    b["mass"] = 1.0
    b["local_inertia"] = scenes.box_inertia(1.0, (0.5, 0.5, 0.5))
    b["transform"][:, [0, 4, 8]] = 1.0
    b["transform"][:, 9] = 0.99 * np.arange(n)
    b["transform"][:, 10] = 0.49
    bodies = np.concatenate([np.concatenate([scenes._plane_body(0), b]) for _ in range(worlds)])
    bodies["world"] = np.repeat(np.arange(worlds), n + 1)
    shapes = [dict(scenes.PLANE), {"type": _abi.SHAPE_BOX, "params": (0.5, 0.5, 0.5, 0.0), "points": None}]
    return scenes.Scene("rows", 1.0 / 60.0, 1, {"gravity": (0.0, -9.81, 0.0)}, shapes, bodies,
                        world_of_body=bodies["world"].astype(np.int32))


@pytest.mark.parametrize("worlds,iterations", [(120, 511), (120, 512), (120, 60000)])   # 360 pieces of 86 bodies
def test_many_iterations(gpu_lib, worlds, iterations):
    n = 257
    sc = _rows(worlds, n)
    flow = gpu_lib.GpuWorld(sc, config=_abi.default_config(**dict(sc.config, num_iterations=iterations)))
    ref = gpu_lib.GpuWorld(sc, config=_abi.default_config(**dict(sc.config, num_iterations=iterations, solver_smem_bodies=1)))
    flow.step(sc.dt)
    ref.step(sc.dt)
    s = flow.get_state()
    assert not H.compare_state(s, ref.get_state())
    assert not H.compare_manifolds(flow.get_manifolds(), ref.get_manifolds())
    for f in H.STATE_COPY:
        a = s[f].reshape((worlds, n + 1) + s[f].shape[1:])
        assert np.all(a == a[:1])
    assert flow.counters()["solver_rows"] > 0
    flow.close()
    ref.close()
