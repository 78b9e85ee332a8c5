"""Gradients of a large batch against the same batch in tiles of 64 samples summed in 64 bits.  The number of
samples is a power of two, so the tiles' roundings to bfloat16 are the same in both, and what differs is
the sum over tiles.  A weight's sum is some 16,384 / 304 additions in a block and one of 304 blocks to
memory: up to 360 roundings to nearest, each at most 2^-25 of a partial sum, of either sign, sqrt(360)
2^-25 / sqrt(3) = 3e-7 for one weight.  That bounds the signed mean as though all weights erred
together; sums cut towards zero are off by 3e-6, all of one sign."""
import numpy as np
import pytest

import mlp_ref as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bias", [0.0, 1.5])
def test_sum_over_tiles(gpu_lib, bias):
    from jbgpu.lib import Mlp
    n, tile = 1 << 20, 64
    rng = np.random.default_rng(n)
    m = Mlp(seed=5)
    m.set_params((rng.standard_normal(R.N_PARAM) * 0.2).astype(np.float32),
                 np.concatenate([rng.standard_normal(R.N_IN) * 0.1, rng.uniform(0.5, 2.0, R.N_IN),
                                 rng.standard_normal(R.N_OUT) * 0.1, rng.uniform(0.5, 2.0, R.N_OUT), [1.0]]).astype(np.float32))
    x = rng.standard_normal((n, R.N_IN)).astype(np.float32)
    t = (rng.standard_normal((n, R.N_OUT)) + bias).astype(np.float32)
    g, loss = m.gradients(x, t)
    want, want_loss = np.zeros(R.N_PARAM), 0.0
    for k in range(0, n, tile):
        gt, lt = m.gradients(x[k: k + tile], t[k: k + tile])
        want += gt
        want_loss += lt
    want *= tile / n
    want_loss *= tile / n
    err = g - want
    assert abs(np.sum(err * np.sign(want))) <= 3e-7 * np.sum(np.abs(want))
    assert abs(loss - want_loss) <= 1e-5 * want_loss
    m.close()
