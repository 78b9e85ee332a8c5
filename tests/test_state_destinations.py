"""get_state into arrays that lie behind one another without being one allocation: pinned memory registered
piece by piece.  The fields arrive as they do in separate arrays."""
import ctypes as C
import mmap

import numpy as np
import pytest

import harness as H
from jbgpu import _abi, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pinned", ["all", "first", "alternate", "none"])
def test_adjacent_arrays_registered_apart(gpu_lib, pinned):
    torch = pytest.importorskip("torch")
    rt = torch.cuda.cudart()
    n = mmap.PAGESIZE // 4                   # every field is a whole number of pages
    b = scenes._bodies(n)
    rng = np.random.Generator(np.random.PCG64(1))
    b["mass"] = 1.0
    b["local_inertia"] = 0.1
    b["linear_velocity"] = rng.normal(0.0, 1.0, (n, 3))
    scenes._set_transforms(b, scenes.random_rotations(rng, n), rng.uniform(-50.0, 50.0, (n, 3)))
    sc = scenes.Scene("state", 1.0 / 60.0, 1, {"gravity": (0.0, -9.81, 0.0)},
                      [{"type": _abi.SHAPE_SPHERE, "params": (0.3, 0.0, 0.0, 0.0), "points": None}], b)
    g = gpu_lib.GpuWorld(sc)
    for _ in range(3):
        g.step(sc.dt)
    ref = g.get_state()
    page = mmap.PAGESIZE
    words = [w for w, _ in _abi.STATE_FIELDS.values()]
    mem = mmap.mmap(-1, 4 * n * sum(words) + page)
    whole = np.frombuffer(mem, np.uint8)
    at, st, out, held = whole.ctypes.data, _abi.State(), {}, []
    offset = 0
    for k, (name, (w, dt)) in enumerate(_abi.STATE_FIELDS.items()):
        size = 4 * n * w
        a = whole[offset: offset + size].view(dt)
        out[name] = a.reshape(n, w) if w > 1 else a
        setattr(st, name, _abi._ptr(out[name], _abi.i32p if dt == np.int32 else _abi.f32p))
        if pinned == "all" or (pinned == "first" and k == 0) or (pinned == "alternate" and k % 2):
            assert int(rt.cudaHostRegister(at + offset, size, 0)) == 0
            held.append(at + offset)
        offset += size
    try:
        gpu_lib.check(gpu_lib.lib().jbgpu_world_get_state(g.h, C.byref(st)))
    finally:
        for p in held:
            rt.cudaHostUnregister(p)
    assert st.n_bodies == n
    assert not H.compare_state(ref, out)
    assert np.array_equal(ref["island_tag"], out["island_tag"])
    g.close()
