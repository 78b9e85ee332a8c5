"""Worlds solved colour by colour, a block each, with velocities in shared memory (a kinematic body with
mass keeps a batch off the flow solver), against global memory (solver_smem_bodies=1) and narrower
blocks: equal bit for bit.  Worlds of one body to more than a colour's 384 threads hold."""
import numpy as np
import pytest

import harness as H
from jbgpu import _abi, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("worlds,nmin,nmax", [(1, 5, 6), (3, 1, 20), (24, 16, 300), (2, 1900, 2040)])
def test_same_in_shared_and_global_memory(gpu_lib, worlds, nmin, nmax):
    sc = scenes.batched_worlds(worlds, seed=worlds, nmin=nmin, nmax=nmax)
    k = len(sc.bodies) - 1
    sc.bodies["collision_flags"][k] |= _abi.CF_KINEMATIC_OBJECT   # keeping its mass
    sc.bodies["transform"][k, 9:] = (300.0, 300.0, 300.0)
    runs = [gpu_lib.GpuWorld(sc, config=_abi.default_config(**dict(sc.config, **kn)))
            for kn in ({}, {"solver_smem_bodies": 1}, {"solver_threads": 128})]
    for step in range(200):
        for g in runs:
            g.step(sc.dt)
        if step % 50 == 49:
            a = runs[0].get_state()
            assert np.all(np.isfinite(a["transform"]))
            for g in runs[1:]:
                assert not H.compare_state(a, g.get_state()), step
                assert not H.compare_manifolds(runs[0].get_manifolds(), g.get_manifolds()), step
                for key in ("solver_rows", "colours", "solver_iterations", "status_flags"):
                    assert runs[0].counters()[key] == g.counters()[key], (step, key)
    assert nmax < 20 or runs[0].counters()["solver_rows"] > 0
    for g in runs:
        g.close()
