"""Colourings that turn to the claim passes in the middle of a launch (a row of touching boxes longer than
the passes' limit, beside worlds and parts that need none), while another world steps on its own stream,
so that blocks start late: state, order and counts equal those of a quiet run bit for bit, and the batch's
the oracle's."""
import threading

import numpy as np
import pytest

import harness as H
import pyoracle
from jbgpu import _abi, scenes

pytestmark = pytest.mark.gpu
CONFIG = {"gravity": (0.0, -9.81, 0.0), "num_iterations": 4}
SHAPES = [dict(scenes.PLANE), {"type": _abi.SHAPE_BOX, "params": (0.5, 0.5, 0.5, 0.0), "points": None}]


def _boxes(pos):
    b = scenes._bodies(len(pos))
    b["shape"] = 1
    b["mass"] = 1.0
    b["local_inertia"] = scenes.box_inertia(1.0, (0.5, 0.5, 0.5))
    b["transform"][:, [0, 4, 8]] = 1.0
    b["transform"][:, 9:] = np.asarray(pos, np.float32)
    return b


def _row(n, z=0.0):
    return [(0.99 * k, 0.49, z) for k in range(n)]


def _stacks(n, z0):
    return [(1.5 * (k // 3 % 20), 0.49 + 0.99 * (k % 3), z0 + 1.5 * (k // 60)) for k in range(n)]


def _batch(worlds=40):
    parts = []
    for w in range(worlds):
        b = np.concatenate([scenes._plane_body(0), _boxes(_row(120) if w % 13 == 5 else _stacks(24 + 3 * w, 0.0))])
        b["world"] = w
        parts.append(b)
    bodies = np.concatenate(parts)
    return scenes.Scene("rows_and_stacks", 1.0 / 60.0, 1, CONFIG, SHAPES, bodies, world_of_body=bodies["world"].astype(np.int32))


def _one_world():
    return scenes.Scene("row_among_stacks", 1.0 / 60.0, 1, CONFIG, SHAPES,
                        np.concatenate([scenes._plane_body(0), _boxes(_row(150) + _stacks(2400, 3.0))]))


def _run(gpu_lib, sc, steps):
    g = gpu_lib.GpuWorld(sc)
    out = []
    for _ in range(steps):
        g.step(sc.dt)
        c = g.counters()
        out.append((g.get_state(), g.solver_order(), [c[k] for k in ("colours", "solver_rows", "cut_manifolds", "status_flags")]))
    g.close()
    return out


@pytest.mark.parametrize("make", [_batch, _one_world])
def test_same_beside_another_stream(gpu_lib, oracle_lib, make):
    sc, steps = make(), 8
    quiet = _run(gpu_lib, sc, steps)
    if make is _batch:
        o = pyoracle.OracleWorld(sc, order_mode=pyoracle.ORDER_COLOUR)
        for k in range(steps):
            o.step(sc.dt)
            assert not H.compare_state(quiet[k][0], o.get_state()), k
    other = scenes.boxes_on_plane(1500, seed=3, region=(12.0, 20.0, 12.0), y0=0.5)
    stop, failed = threading.Event(), []

    def neighbour():
        try:
            w = gpu_lib.GpuWorld(other)
            while not stop.is_set():
                w.step(other.dt)
            w.close()
        except Exception as e:   # pragma: no cover
            failed.append(e)

    t = threading.Thread(target=neighbour)
    t.start()
    try:
        runs = [_run(gpu_lib, sc, steps) for _ in range(6)]
    finally:
        stop.set()
        t.join()
    assert not failed
    for run in runs:
        for k in range(steps):
            assert not H.compare_state(quiet[k][0], run[k][0]), k
            assert np.array_equal(quiet[k][1], run[k][1]) and quiet[k][2] == run[k][2], k
    assert quiet[-1][2][1] > 0 and quiet[-1][2][3] == 0
