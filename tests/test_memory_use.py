"""Device memory that reading a world takes: transforms stage twelve words a body, not a whole state."""
import numpy as np
import pytest

from jbgpu import _abi, scenes

pytestmark = pytest.mark.gpu
MB = 1 << 20


def _free():
    torch = pytest.importorskip("torch")
    return torch.cuda.mem_get_info()[0]


def test_transforms_stage_twelve_words_a_body(gpu_lib):
    n = 300000
    b = scenes._bodies(n)
    b["transform"][:, 9] = np.arange(n)
    sc = scenes.Scene("rest", 1.0 / 60.0, 1, {"gravity": (0.0, 0.0, 0.0)},
                      [{"type": _abi.SHAPE_SPHERE, "params": (0.3, 0.0, 0.0, 0.0), "points": None}], b)
    g = gpu_lib.GpuWorld(sc)
    before = _free()
    assert np.array_equal(g.get_transforms()[:, 9], np.arange(n, dtype=np.float32))
    assert before - _free() <= 48 * n + 4 * MB
    t = g.get_state()["transform"]                                     # the larger stage, then transforms again
    assert np.array_equal(t, g.get_transforms())
    g.close()
