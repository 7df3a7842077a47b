"""Closest-hit and occlusion launches around the counts at which they change
how many walks a warp takes: the same radiance as in a launch of full warps on
both passes, bit for bit."""
import numpy as np
import pytest

import bevy_penumbra_b200 as bp
from tests.helpers import empty_device, from_device, packed, to_device
from tests.test_gpu_radiance import random_rays

pytestmark = pytest.mark.gpu

# 148 SMs x 16 blocks x 4 warps = 9472 warps: closest hits take 4 walks per
# warp up to 37,888 rays and 8 up to 75,776; occlusion, in half of the warps,
# up to 16 walks for 75,776 queries, which this many rays exceed.
FULL = 160_000


def radiance(n):
    rays = random_rays(FULL, (-7.0, 0.1, -7.0), (7.0, 4.0, 7.0), seed=13)
    ctx = bp.LuxContext()
    scene = bp.GpuScene(ctx, packed("atrium65536"))
    d_rays, out = to_device(rays), empty_device(FULL * 16)
    settings = bp.RadianceCascades(frame_index=3, emissive_samples=4).sanitized()
    bp.interval_radiance(ctx, scene, settings, d_rays.data_ptr(), n, out.data_ptr())
    return from_device(out, np.uint32, (FULL, 4))[:n]


@pytest.fixture(scope="module")
def full():
    return radiance(FULL)


@pytest.mark.parametrize("n", [1, 37_887, 37_888, 37_889, 75_776, 75_777, 120_001])
def test_radiance_at_the_edges_of_each_kind_of_launch(full, n):
    np.testing.assert_array_equal(radiance(n), full[:n])
