"""Learned radiance cache: encoded rows of ragged sample counts bit for bit,
and one Adam step at the smallest table."""
import numpy as np
import pytest

import bevy_penumbra_b200 as bp
from tests.helpers import empty_device, from_device, to_device
from tests.test_gpu_cache import bf16_round, field, make_cache, random_samples
from tests.test_gpu_cache_grad import corners

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,levels,table,offset", [(1, 16, 14, 0), (31, 5, 8, 4), (33, 16, 10, 4), (130, 1, 8, 0)])
def test_encoded_features_match_the_corner_sums(n, levels, table, offset):
    """Features are the corners' weighted sums in corner order, in FP32,
    rounded to BF16; samples need only be 4-byte aligned."""
    ctx = bp.LuxContext()
    cache = make_cache(ctx, levels=levels, log2_table=table)
    s = random_samples(n, 3 + n)
    s["position"][0] = (2.0, -2.0, 5.0)  # on and past the box's faces
    raw = to_device(np.concatenate([np.zeros(offset, np.uint8), s.view(np.uint8).reshape(-1)]))
    out = empty_device(n * 128)
    cache.encode(raw.data_ptr() + offset, n, out.data_ptr())
    ctx.synchronize()
    got = from_device(out, np.uint16, (n, 64))
    idx, wts = corners(cache, s)
    rows = bf16_round(cache.table().reshape(-1, 2)).numpy()
    want = np.zeros((n, 32), np.float32)
    for c in range(2):
        acc = np.zeros((n, levels), np.float32)
        for k in range(8):
            acc = acc + wts[:, :, k] * rows[idx[:, :, k], c]
        want[:, c:2 * levels:2] = acc
    bits = (bf16_round(want).numpy().view(np.uint32) >> 16).astype(np.uint16)
    np.testing.assert_array_equal(got[:, :32], bits)
    assert (got[:, 54] == 0x3f80).all() and (got[:, 55:] == 0).all()


@pytest.mark.parametrize("n,levels", [(128, 1), (300, 3)])
def test_first_adam_step_moves_reached_entries_by_the_rate(n, levels):
    """Adam's first update is the learning rate against the gradient's sign
    (to FP32 rounding of the bias corrections); other entries stay."""
    ctx = bp.LuxContext()
    cache = make_cache(ctx, levels=levels, log2_table=8, batch=512, learning_rate=1e-2)
    s = random_samples(n, 7)
    t = field(s)
    d_s, d_t = to_device(s), to_device(t)
    _, g = cache.gradients(d_s.data_ptr(), d_t.data_ptr(), n)
    g, before = g.reshape(-1), cache.table().reshape(-1).copy()
    cache.train(d_s.data_ptr(), d_t.data_ptr(), n)
    step = cache.table().reshape(-1) - before
    assert cache.stats().error_flags == 0
    np.testing.assert_array_equal(step[g == 0.0], 0.0)
    clear = np.abs(g) > 1e-3 * np.abs(g).max()  # the sum's order cannot turn these
    np.testing.assert_allclose(step[clear], -1e-2 * np.sign(g[clear]), rtol=1e-4)
