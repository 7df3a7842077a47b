"""Scene words whose local_from_world rows are not the inverse of their
world_from_local rows: the walk follows local_from_world alone, as the oracle's
does, whatever tree it takes."""
import numpy as np
import pytest

import bevy_penumbra_b200 as bp
import oracle
from tests.helpers import EMPTY, empty_device, from_device, to_device
from tests.test_gpu_far_rays import grid_scene, rays_to

pytestmark = pytest.mark.gpu


# Shifts of the local ray: an inverse in single precision, and one that is off
# by a fifth of a triangle.
@pytest.mark.parametrize("shift", [1e-6, 2e-3])
def test_rows_that_are_not_inverses(shift):
    packed, m = grid_scene((0.5, 0.25, -0.5))
    words = packed.scene_words.copy()
    for slot in range(len(packed.instance_order)):
        first = int(words[0, 1]) + 9 * slot
        words[first:first + 3].view(np.float32)[:, 3] += np.float32(shift)
    rays = rays_to(m, 3.0, 4000, 3)
    want, _ = oracle.OracleScene(words, packed.geometry_words, packed.lights).trace_rays(rays)
    assert np.mean(want["triangle"] != EMPTY) > 0.9
    ctx = bp.LuxContext()
    scene = bp.GpuScene(ctx, bp.PackedScene(words, packed.geometry_words, packed.lights))
    d_rays, d_hits = to_device(rays), empty_device(len(rays) * bp.HIT_DTYPE.itemsize)
    bp.trace_rays(ctx, scene, d_rays.data_ptr(), len(rays), d_hits.data_ptr())
    got = from_device(d_hits, bp.HIT_DTYPE, (len(rays),))
    np.testing.assert_array_equal(got["triangle"], want["triangle"])
    np.testing.assert_array_equal(got["distance"].view(np.uint32), want["distance"].view(np.uint32))
