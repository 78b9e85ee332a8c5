"""Selection and solver preparation by one block (up to 4,096 bodies and a pair capacity of 2,048) and by
their launches, on worlds that start on one side of the line and grow past it: state, colours and counts
equal the oracle's in the GPU's manifold order, closed loop, through falling, resting and sleeping."""
import numpy as np
import pytest

import harness as H
import pyoracle
from jbgpu import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,side,steps", [(1, 3.0, 30), (20, 3.0, 150), (120, 4.0, 60), (330, 6.0, 60), (450, 7.0, 60),
                                          (900, 9.0, 40)])
def test_same_as_the_oracle(gpu_lib, oracle_lib, n, side, steps):
    sc = scenes.boxes_on_plane(n, seed=n, region=(side, 2.0 + n / (side * side) * 2.0, side), y0=0.5)
    g = gpu_lib.GpuWorld(sc)
    o = pyoracle.OracleWorld(sc, order_mode=pyoracle.ORDER_COLOUR)
    for k in range(steps):
        g.step(sc.dt)
        o.step(sc.dt)
        if k % 10 == 9:
            a, b = g.counters(), o.counters()
            for key in ("pairs", "manifolds", "contacts", "islands", "solver_manifolds", "solver_rows", "colours"):
                assert a[key] == b[key], (k, key, a[key], b[key])
            assert not H.compare_state(g.get_state(), o.get_state()), k
    assert n == 1 or a["contacts"] > 0
    g.close()
