"""Jointed worlds whose kinematic body keeps its mass: joints and contacts act on its velocity while a step
is solved (the next saveKinematicState sets it again), and contacts see what the joints did to it.  A
world of one part and the same world twice in a batch (two parts) solve the same bit for bit; so does a
world whose kinematic body has no mass, and one without a contact on it."""
import numpy as np
import pytest

import harness as H
from jbgpu import _abi, scenes

pytestmark = pytest.mark.gpu


def _scene(worlds, mass, box):
    """Per world: a kinematic plate, a link hanging from it on a ball joint and swinging, and (box) a box
    dropped onto the plate.  One manifold and one joint on the plate, so that nothing in a colour shares it."""
    shapes = [dict(scenes.PLANE), {"type": _abi.SHAPE_BOX, "params": (1.0, 0.2, 1.0, 0.0), "points": None},
              {"type": _abi.SHAPE_BOX, "params": (0.15, 0.45, 0.15, 0.0), "points": None},
              {"type": _abi.SHAPE_BOX, "params": (0.3, 0.3, 0.3, 0.0), "points": None}]
    bodies, joints = [], []
    for w in range(worlds):
        b = scenes._bodies(3 if box else 2)
        b["shape"][:2] = (1, 2)
        b["mass"][:2] = (mass, 2.0)
        b["collision_flags"][0] = _abi.CF_KINEMATIC_OBJECT
        b["activation_state"][0] = _abi.DISABLE_DEACTIVATION
        if mass:
            b["local_inertia"][0] = scenes.box_inertia(mass, (1.0, 0.2, 1.0))
        b["local_inertia"][1] = scenes.box_inertia(2.0, (0.15, 0.45, 0.15))
        b["linear_velocity"][1] = (1.5, 0.0, 0.7)
        b["transform"][:, [0, 4, 8]] = 1.0
        b["transform"][:2, 9:] = ((0.0, 4.0, 0.0), (0.0, 2.8, 0.0))
        if box:
            b["shape"][2] = 3
            b["mass"][2] = 1.0
            b["local_inertia"][2] = scenes.box_inertia(1.0, (0.3, 0.3, 0.3))
            b["transform"][2, 9:] = (-0.5, 4.52, 0.1)
        first = sum(len(x) for x in bodies)
        joints.append({"a": first + 2, "b": first + 1, "pivot_a": (0.0, 0.5, 0.0), "pivot_b": (0.0, -0.7, 0.0)})
        bodies.append(np.concatenate([scenes._plane_body(0), b]))
        bodies[-1]["world"] = w
    kw = {"world_of_body": np.repeat(np.arange(worlds, dtype=np.int32), len(bodies[0]))} if worlds > 1 else {}
    return scenes.Scene("kinematic_joint", 1.0 / 60.0, 1, {"gravity": (0.0, -9.81, 0.0), "num_iterations": 10}, shapes,
                        np.concatenate(bodies), meta={"joints": joints}, **kw)


@pytest.mark.parametrize("mass,box", [(5.0, True), (0.5, True), (5.0, False), (0.0, True)])
def test_alone_same_as_in_a_batch(gpu_lib, mass, box):
    one, two = _scene(1, mass, box), _scene(2, mass, box)
    n = len(one.bodies)
    g, b = gpu_lib.GpuWorld(one), gpu_lib.GpuWorld(two)
    touched = 0
    for k in range(30):
        g.step(one.dt)
        b.step(two.dt)
        touched += g.counters()["solver_manifolds"]
        s, t = g.get_state(), b.get_state()
        for half in (slice(0, n), slice(n, 2 * n)):
            assert not H.compare_state(s, {f: t[f][half] for f in H.STATE_COPY}), k
    assert (touched > 0) == box
    g.close()
    b.close()
