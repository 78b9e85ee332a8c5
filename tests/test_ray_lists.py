"""The candidate lists of large ray batches: no more entries a ray than the world has bodies, half as many as
often as the device has no room (the rule compiled for the host, with an allocator that refuses), and rays
on worlds of a few bodies, whose lists are that short, equal to the oracle's."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from jbgpu import _abi, scenes
from jbgpu._build import CSRC

MAIN = r"""
#include <cstdio>
#include <cstdlib>
#include "ray_lists.cuh"
int main(int argc, char** argv) {   // rays bodies held room -> entries a ray, entries allocated, tries
    const int rays = atoi(argv[1]), bodies = atoi(argv[2]);
    size_t held = strtoull(argv[3], nullptr, 10);
    const size_t room = strtoull(argv[4], nullptr, 10);
    int tries = 0;
    const int cap = jbg::ray_list_fit(rays, bodies, held, [&](size_t n) {
        tries++;
        held = n <= room ? n : 0;
        return held != 0;
    });
    printf("%d %zu %d\n", cap, held, tries);
}
"""
BIG = 1 << 40


@pytest.fixture(scope="module")
def fit(tmp_path_factory):
    d = tmp_path_factory.mktemp("ray_lists")
    (d / "main.cpp").write_text(MAIN)
    subprocess.run([shutil.which("g++") or "c++", "-std=c++17", "-x", "c++", "-I", CSRC, str(d / "main.cpp"), "-o", str(d / "fit")],
                   check=True)
    return lambda *a: tuple(int(x) for x in subprocess.check_output([str(d / "fit")] + [str(x) for x in a]).split())


@pytest.mark.parametrize("rays,bodies,held,room,want", [
    (200000, 100000, 0, BIG, (256, 200000 * 256, 1)),
    (200000, 61, 0, BIG, (61, 200000 * 61, 1)),
    (200000, 1, 0, BIG, (1, 200000, 1)),
    (1 << 20, 1000, 0, BIG, (64, 1 << 26, 1)),
    (1 << 24, 1000, 0, BIG, (8, 1 << 27, 1)),
    (1 << 24, 5, 0, BIG, (5, 5 << 24, 1)),
    (100, 1000, 25600, 0, (256, 25600, 0)),          # what there is suffices
    (100, 1000, 25599, 1 << 30, (256, 25600, 1)),
    (100, 1000, 0, 25599, (128, 12800, 2)),          # no room: half
    (100, 1000, 0, 1000, (8, 800, 6)),
    (100, 61, 0, 200, (1, 100, 6)),
    (100, 61, 50, 99, (0, 0, 6)),                    # not even one entry a ray
])
def test_entries_a_ray(fit, rays, bodies, held, room, want):
    assert fit(rays, bodies, held, room) == want


def _free():
    torch = pytest.importorskip("torch")
    return torch.cuda.mem_get_info()[0]


@pytest.mark.gpu
def test_memory_of_a_batch_in_a_small_world(gpu_lib):
    sc = scenes.small_mixed(60, seed=2)
    n, bodies = 200000, len(sc.bodies)
    g = gpu_lib.GpuWorld(sc)
    up = np.tile(np.float32([0.0, 1000.0, 0.0]), (n, 1))
    g.ray_test(up[:20000], up[:20000] + np.float32([0.0, 1.0, 0.0]))   # code and first buffers
    before = _free()
    h = g.ray_test(up, up + np.float32([0.0, 1.0, 0.0]))
    assert np.all(h["body"] == -1)
    # lists of 8 bytes an entry, rays and hits (60 bytes), counts, offsets, keys, scan (24 bytes)
    assert before - _free() <= n * (8 * bodies + 60 + 24) + (16 << 20)
    g.close()


@pytest.mark.gpu
@pytest.mark.parametrize("bodies", [1, 2, 5, 9])
def test_worlds_of_a_few_bodies(gpu_lib, oracle_lib, bodies):
    import pyoracle
    b = scenes._bodies(bodies)
    b["transform"][:, 9:] = np.linspace(0.0, 1.0, 3 * bodies).reshape(bodies, 3)
    sc = scenes.Scene("few", 1.0 / 60.0, 1, {}, [{"type": _abi.SHAPE_SPHERE, "params": (1.0, 0.0, 0.0, 0.0), "points": None}], b)
    rng = np.random.Generator(np.random.PCG64(bodies))
    frm, to = (rng.uniform(-3.0, 4.0, (9000, 3)).astype(np.float32) for _ in range(2))
    g = gpu_lib.GpuWorld(sc)
    want = pyoracle.OracleWorld(sc).ray_test(frm, to)
    assert np.any(want["body"] >= 0)
    assert np.array_equal(want.view(np.uint8), g.ray_test(frm, to).view(np.uint8))
    g.close()
