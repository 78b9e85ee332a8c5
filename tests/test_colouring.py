"""The colouring's two paths against the oracle's claim passes, closed loop and bit for bit, around
the limits that choose between them: rows of touching boxes in index order, whose claim passes grow
with the row's length (past 16 a colour stays unfinished, which only the claim passes give), and a
dynamic plate carrying more boxes than a body's candidate list holds."""
import numpy as np
import pytest

import harness as H
import pyoracle
from jbgpu import _abi, scenes

pytestmark = pytest.mark.gpu
CONFIG = {"gravity": (0.0, -9.81, 0.0), "num_iterations": 10}


def _scene(name, half, pos, mass):
    shapes = [dict(scenes.PLANE)] + [{"type": _abi.SHAPE_BOX, "params": (*h, 0.0), "points": None} for h in half]
    b = scenes._bodies(len(pos))
    b["shape"] = [1 if len(half) == 1 or k == 0 else 2 for k in range(len(pos))]
    b["mass"] = mass
    for k in range(len(pos)):
        b["local_inertia"][k] = scenes.box_inertia(b["mass"][k], half[b["shape"][k] - 1])
    b["transform"][:, 9:] = np.asarray(pos, np.float32)
    return scenes.Scene(name, 1.0 / 60.0, 0, CONFIG, shapes, np.concatenate([scenes._plane_body(0), b]))


def _row(n):
    return _scene("row_%d" % n, [(0.5, 0.5, 0.5)], [(0.99 * k, 0.49, 0.0) for k in range(n)], 1.0)


def _plate(n):
    side = int(np.ceil(np.sqrt(n)))
    boxes = [(0.7 * (k % side) - 0.35 * side, 0.69, 0.7 * (k // side) - 0.35 * side) for k in range(n)]
    return _scene("plate_%d" % n, [(0.4 * side + 1.0, 0.25, 0.4 * side + 1.0), (0.2, 0.2, 0.2)], [(0.0, 0.24, 0.0)] + boxes,
                  [50.0] + [0.5] * n)


CASES = {"row_%d" % n: (_row, n) for n in (2, 16, 31, 33, 35, 48, 120)}
CASES.update({"plate_%d" % n: (_plate, n) for n in (30, 31, 32, 33, 60, 70)})


@pytest.mark.parametrize("name", list(CASES))
def test_same_colours_as_claim_passes(gpu_lib, oracle_lib, name):
    make, n = CASES[name]
    sc = make(n)
    g = gpu_lib.GpuWorld(sc)
    o = pyoracle.OracleWorld(sc, order_mode=pyoracle.ORDER_COLOUR)
    for k in range(6):
        g.step(sc.dt)
        o.step(sc.dt)
        assert g.counters()["solver_manifolds"] > 0
        assert g.counters()["colours"] == o.counters()["colours"], k
        assert not H.compare_state(g.get_state(), o.get_state()), k
    g.close()
