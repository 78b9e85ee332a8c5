"""What test_flow_solver.py compares: each of its worlds runs the flow solver, and its reference world the
colour-by-colour solver (told apart by the launches of the solve, which lays out no slots for the flow
solver) - except the world of one body, whose part no solver_smem_bodies is below; that one is compared
with the oracle."""
import numpy as np
import pytest

import harness as H
import pyoracle
from jbgpu import _abi
from test_flow_solver import CASES

pytestmark = pytest.mark.gpu
STAGES = (_abi.STAGE_APPLY_GRAVITY, _abi.STAGE_PREDICT, _abi.STAGE_AABB, _abi.STAGE_PAIRS, _abi.STAGE_NARROWPHASE,
          _abi.STAGE_ISLANDS)


def _solve_launches(gpu_lib, sc, steps, **config):
    g = gpu_lib.GpuWorld(sc, config=_abi.default_config(**dict(sc.config, **config)))
    for _ in range(steps):
        g.step(sc.dt)
    for stage in STAGES:
        g.stage(stage, sc.dt)
    before = gpu_lib.launch_count()
    g.stage(_abi.STAGE_SOLVE, sc.dt)
    n = gpu_lib.launch_count() - before
    rows = g.counters()["solver_rows"]
    g.close()
    return n, rows


@pytest.mark.parametrize("name", [k for k in CASES if k != "one_body"])
def test_two_solvers_are_compared(gpu_lib, name):
    make, knobs, steps = CASES[name]
    sc = make()
    flow, rows = _solve_launches(gpu_lib, sc, steps, **knobs)
    ref, _ = _solve_launches(gpu_lib, sc, steps, solver_smem_bodies=1, **knobs)
    assert rows > 0
    assert flow + 2 <= ref                      # gather and solve; slots, scan, setup and solve


def test_one_body_same_as_the_oracle(gpu_lib, oracle_lib):
    sc = CASES["one_body"][0]()
    g = gpu_lib.GpuWorld(sc)
    o = pyoracle.OracleWorld(sc, order_mode=pyoracle.ORDER_COLOUR)
    for k in range(120):                        # it lands after some fifty steps
        g.step(sc.dt)
        o.step(sc.dt)
        assert not H.compare_state(g.get_state(), o.get_state()), k
    assert g.counters()["solver_rows"] == o.counters()["solver_rows"] > 0
    g.close()
