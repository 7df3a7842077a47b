"""Short trace launches take fewer walks per warp: every count's hits and
radiance are those of the same rays in a launch of full warps, bit for bit."""
import numpy as np
import pytest

import bevy_penumbra_b200 as bp
from tests.helpers import empty_device, from_device, packed, to_device
from tests.test_gpu_radiance import random_rays

pytestmark = pytest.mark.gpu

FULL = 50000  # more rays than a short launch takes on any of its paths


def run(n, any_hit):
    """Hits or (any_hit None) interval radiance of the first n rays."""
    rays = random_rays(FULL, (-7.0, 0.1, -7.0), (7.0, 4.0, 7.0), seed=9)
    ctx = bp.LuxContext()
    scene = bp.GpuScene(ctx, packed("atrium65536"))
    d_rays = to_device(rays)
    if any_hit is None:
        out = empty_device(FULL * 16)
        settings = bp.RadianceCascades(frame_index=3, emissive_samples=4).sanitized()
        bp.interval_radiance(ctx, scene, settings, d_rays.data_ptr(), n, out.data_ptr())
        ctx.synchronize()
        return from_device(out, np.uint32, (FULL, 4))[:n]
    out = empty_device(FULL * bp.HIT_DTYPE.itemsize)
    bp.trace_rays(ctx, scene, d_rays.data_ptr(), n, out.data_ptr(), any_hit=any_hit)
    return from_device(out, np.uint32, (FULL, bp.HIT_DTYPE.itemsize // 4))[:n]


@pytest.fixture(scope="module")
def full():
    return {any_hit: run(FULL, any_hit) for any_hit in (False, True, None)}


# 148 SMs x 28 warps x 4 and x 8 rays: the last launches of each kind.
@pytest.mark.parametrize("n", [1, 3, 5, 513, 16576, 16577, 33152, 33153])
def test_counts_at_the_edges_of_each_kind_of_launch(full, n):
    for any_hit in (False, True, None):
        np.testing.assert_array_equal(run(n, any_hit), full[any_hit][:n], err_msg=str(any_hit))
