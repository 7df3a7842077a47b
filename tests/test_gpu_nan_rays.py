"""Caller rays with a NaN bound hit nothing, as in the oracle."""
import numpy as np
import pytest

import bevy_penumbra_b200 as bp
import oracle
from tests.helpers import EMPTY
from tests.test_gpu_flat import POSES, cornell_with, trace
from tests.test_gpu_radiance import random_rays

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pose", ["rotated", "ill-sheared"])  # the flattened tree, the two-level walk
@pytest.mark.parametrize("far", [False, True])
@pytest.mark.parametrize("bound", ["tmin", "limit"])
def test_rays_with_a_nan_bound_hit_nothing(pose, far, bound):
    packed = cornell_with(POSES[pose])
    rays = random_rays(300, (-0.95, 0.05, -0.95), (0.95, 1.95, 0.95), seed=4)
    if far:
        rays["origin"] += np.float32(100.0)
        rays["direction"] = np.float32([0.0, 1.0, 0.0]) - rays["origin"]
    rays[bound][::3] = np.nan
    for any_hit in (False, True):
        cpu, _ = oracle.OracleScene.from_packed(packed).trace_rays(rays, any_hit=any_hit)
        gpu = trace(packed, rays, any_hit)
        np.testing.assert_array_equal(gpu["triangle"] != EMPTY, cpu["triangle"] != EMPTY)
        np.testing.assert_array_equal(gpu["errors"], cpu["errors"])
        if not any_hit or bound == "limit":
            assert np.all(cpu["triangle"][::3] == EMPTY) and np.any(cpu["triangle"] != EMPTY)
