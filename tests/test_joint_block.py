"""Joints solved by one block with the part's velocities in shared memory (the default) against the general
loop on global memory (solver_smem_bodies below the part): every joint kind, joints without contacts, one
link more than a warp, joints and contacts on the same bodies.  Equal bit for bit; the joint tests compare
the default with the oracle."""
import numpy as np
import pytest

import harness as H
from jbgpu import _abi, scenes

pytestmark = pytest.mark.gpu

CASES = {
    "one_hinge": lambda: scenes.hinged_chains(chains=1, links=1, loose=0),
    "hinges_33": lambda: scenes.hinged_chains(chains=1, links=33, loose=0),
    "hinges_and_boxes": lambda: scenes.hinged_chains(chains=5, links=6, loose=25),
    "many_hinges": lambda: scenes.hinged_chains(chains=40, links=8, loose=60),
    "balls": lambda: scenes.jointed_chains(chains=9, links=7, loose=30, seed=4),
    "sixdof": lambda: scenes.sixdof_chains(chains=8, links=4, loose=16, seed=10),
    "cones": lambda: scenes.cone_chains(chains=6, links=5, loose=8, seed=13),
    "sliders": lambda: scenes.slider_rigs(rigs=9, loose=8, seed=15),
}


@pytest.mark.parametrize("name", list(CASES))
def test_same_as_the_general_loop(gpu_lib, name):
    sc = CASES[name]()
    g = gpu_lib.GpuWorld(sc)
    ref = gpu_lib.GpuWorld(sc, config=_abi.default_config(**dict(sc.config, solver_smem_bodies=1)))
    for k in range(50):
        g.step(sc.dt)
        ref.step(sc.dt)
        if k % 10 == 9:
            a = g.get_state()
            assert np.all(np.isfinite(a["transform"]))
            assert not H.compare_state(ref.get_state(), a), k
            assert not H.compare_manifolds(ref.get_manifolds(), g.get_manifolds()), k
    for key in ("solver_rows", "colours", "solver_iterations", "status_flags"):
        assert ref.counters()[key] == g.counters()[key], key
    g.close()
    ref.close()
