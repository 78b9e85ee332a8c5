"""Islands by one block (up to 8,192 bodies and pairs) and by the launch chain, at the edges of the line
between them and of the block: island tags, activation states and counts equal the oracle's
(SimulationIslandManager.java:79-148, DiscreteDynamicsWorld.calculateSimulationIslands)."""
import numpy as np
import pytest

import harness as H
import pyoracle
from jbgpu import _abi, scenes

pytestmark = pytest.mark.gpu


def _chains(n, seed):
    """n spheres on lines in shuffled body order, neighbours touching; every 37th static, some asleep."""
    rng = np.random.Generator(np.random.PCG64(seed))
    shapes = [{"type": _abi.SHAPE_SPHERE, "params": (0.5, 0.0, 0.0, 0.0), "points": None}]
    b = scenes._bodies(n)
    b["shape"] = 0
    b["mass"] = 1.0
    b["local_inertia"] = 0.1
    place = rng.permutation(n)
    b["transform"][:, 9] = 0.95 * (place % 900)
    b["transform"][:, 10] = 3.0 * (place // 900)
    still = place % 37 == 11
    b["mass"][still] = 0.0
    b["local_inertia"][still] = 0.0
    return scenes.Scene("chains", 1.0 / 60.0, 1, {"gravity": (0.0, 0.0, 0.0)}, shapes, b), place


def _least(tags):
    """Each island named by its least body (the oracle names it by its union-find root)."""
    out = tags.copy()
    for t in np.unique(tags[tags >= 0]):
        out[tags == t] = np.nonzero(tags == t)[0][0]
    return out


@pytest.mark.parametrize("n", [1, 2, 33, 1024, 1025, 5000, 8191, 8192, 8193, 9000])
def test_same_islands_as_the_oracle(gpu_lib, oracle_lib, n):
    sc, place = _chains(n, n)
    g = gpu_lib.GpuWorld(sc)
    o = pyoracle.OracleWorld(sc)
    st = g.get_state()
    act = st["activation_state"].copy()
    act[(place // 50) % 3 == 1] = 2                       # ISLAND_SLEEPING
    for w in (g, o):
        w.set_state(dict(activation_state=act, **{k: st[k] for k in ("transform", "linear_velocity", "angular_velocity",
                                                                     "deactivation_time")}))
        for stage in (_abi.STAGE_PREDICT, _abi.STAGE_AABB, _abi.STAGE_PAIRS, _abi.STAGE_NARROWPHASE, _abi.STAGE_ISLANDS):
            w.stage(stage, sc.dt)
    a, b = o.get_state(), g.get_state()
    assert np.array_equal(_least(a["island_tag"]), b["island_tag"])
    assert np.array_equal(a["activation_state"], b["activation_state"])
    for key in ("islands", "manifolds", "contacts"):
        assert o.counters()[key] == g.counters()[key], key
    g.close()
