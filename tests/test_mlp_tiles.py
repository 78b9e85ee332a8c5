"""The network's gradients at the edges of the training kernel's 64-sample tiles and of its grid (blocks
that take several tiles), against the numpy oracle with the kernel's bfloat16 roundings.  Tolerances as
in test_mlp.py's gradient test: a bfloat16 activation that rounds the other way moves single entries by
2^-8, so the whole gradient agrees to 1e-2 relative L2 error and each parameter block to 2e-2; with fewer
than a tile of samples nothing averages such steps out, and the bounds are twice as wide."""
import numpy as np
import pytest

import mlp_ref as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 15, 63, 64, 65, 129, 64 * 304 + 1, 64 * 609])
def test_gradients(gpu_lib, n):
    from jbgpu.lib import Mlp
    rng = np.random.default_rng(n)
    p = (rng.standard_normal(R.N_PARAM) * 0.2).astype(np.float32)
    norm = np.concatenate([rng.standard_normal(R.N_IN) * 0.1, rng.uniform(0.5, 2.0, R.N_IN),
                           rng.standard_normal(R.N_OUT) * 0.1, rng.uniform(0.5, 2.0, R.N_OUT), [1.0]]).astype(np.float32)
    m = Mlp(seed=5)
    m.set_params(p, norm)
    x = rng.standard_normal((n, R.N_IN)).astype(np.float32)
    t = rng.standard_normal((n, R.N_OUT)).astype(np.float32)
    wide = 2.0 if n < 64 else 1.0
    for _ in range(2):                                  # the second call starts from cleared sums
        g, loss = m.gradients(x, t)
        loss_ref, g_ref = R.loss_and_grad(p, norm, x, t, bf16=True)
        assert abs(loss - loss_ref) <= wide * 1e-3 * loss_ref + 1e-6
        assert np.linalg.norm(g - g_ref) <= wide * 1e-2 * np.linalg.norm(g_ref)
        for lo, hi in [(R.OFF_W1, R.OFF_B1), (R.OFF_B1, R.OFF_W2), (R.OFF_W2, R.OFF_B2), (R.OFF_B2, R.OFF_W3),
                       (R.OFF_W3, R.OFF_B3), (R.OFF_B3, R.N_PARAM)]:
            assert np.linalg.norm(g[lo:hi] - g_ref[lo:hi]) <= wide * 2e-2 * np.linalg.norm(g_ref[lo:hi]), (lo, hi)
    m.close()
