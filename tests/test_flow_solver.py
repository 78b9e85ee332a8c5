"""The flow solver (solver_flow.cu) against the colour-by-colour solver on the GPU: both run the same
manifold order, so state and manifolds are equal bit for bit.  solver_smem_bodies below the largest
part keeps a world on the colour-by-colour solver.  The scenes put the flow solver's blocks where they
can go wrong: worlds of one body, of one block and one body more (96 and 97), of many blocks that
exchange velocities, range parts with cut manifolds, parts too large for shared memory (rows and slots
in global memory), groups of 1 to 8 manifolds, blocks of 64 threads, one iteration."""
import numpy as np
import pytest

import harness as H
from jbgpu import _abi, scenes

pytestmark = pytest.mark.gpu


def _boxes(n, side):
    return scenes.boxes_on_plane(n, seed=n, region=(side, 2.0 + n / (side * side) * 2.0, side), y0=0.5)


CASES = {
    "one_body": (lambda: _boxes(1, 3.0), {}, 40),
    "block_96": (lambda: _boxes(96, 5.0), {}, 60),
    "block_97": (lambda: _boxes(97, 5.0), {}, 60),
    "pieces_700": (lambda: _boxes(700, 9.0), {}, 60),
    "pieces_700_64_threads": (lambda: _boxes(700, 9.0), {"solver_threads": 64}, 40),
    "one_iteration": (lambda: _boxes(300, 7.0), {"num_iterations": 1}, 40),
    "mixed_kinds": (lambda: scenes.small_mixed(200, seed=3, region=(7.0, 8.0, 7.0)), {}, 60),
    "worlds": (lambda: scenes.batched_worlds(48, seed=2, nmin=1, nmax=260), {}, 60),
    "range_parts": (lambda: _boxes(2500, 14.0), {}, 50),
    "range_2_parts_far": (lambda: _boxes(3000, 14.0), {"solver_parts": 2}, 50),
    "range_33_parts": (lambda: _boxes(700, 9.0), {"solver_parts": 33}, 50),
    "kinematic": (lambda: scenes.kinematic_platforms(), {}, 60),
}


@pytest.mark.parametrize("name", list(CASES))
def test_same_as_colour_by_colour(gpu_lib, name):
    make, knobs, steps = CASES[name]
    sc = make()
    flow = gpu_lib.GpuWorld(sc, config=_abi.default_config(**dict(sc.config, **knobs)))
    ref = gpu_lib.GpuWorld(sc, config=_abi.default_config(**dict(sc.config, solver_smem_bodies=1, **knobs)))
    for k in range(steps):
        flow.step(sc.dt)
        ref.step(sc.dt)
        if k % 10 == 9 or k == steps - 1:
            a, b = flow.get_state(), ref.get_state()
            assert not H.compare_state(a, b), k
            assert not H.compare_manifolds(flow.get_manifolds(), ref.get_manifolds()), k
            ca, cb = flow.counters(), ref.counters()
            for key in ("solver_rows", "solver_manifolds", "colours", "solver_iterations", "status_flags"):
                assert ca[key] == cb[key], (k, key, ca[key], cb[key])
    assert np.all(np.isfinite(a["transform"]))
    flow.close()
    ref.close()
