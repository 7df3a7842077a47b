"""The mixture of training samples in each batch of a learned-cache frame.  The
samples take their slots in order of arrival, and which arrive first decides
what the network has learned last."""
import numpy as np
import pytest

import bevy_penumbra_b200 as bp
from tests.helpers import empty_device, from_device, packed, to_device
from tests.test_gpu_batch import floor_receivers

pytestmark = pytest.mark.gpu

# Mean prediction (over rgb) at the points below after two frames of sixteen
# batches each: the mean of ten runs of the selection whose threads sum their
# ray's samples one after another.
PREDICTED = np.array([
    0.1407, 0.0626, 0.1425, 0.0713, 0.0763, 0.0837, 0.0813, 0.0691, 0.0868, 0.0734,
    0.0724, 0.0602, 0.0631, 0.0448, 0.0781, 0.0707, 0.0456, 0.0632, 0.0519, 0.0710,
    0.1165, 0.1151, 0.0270, 0.0705, 0.1330, 0.0480, 0.0819, 0.0463, 0.1185, 0.0862,
    0.0592, 0.0624, 0.0680, 0.0372, 0.1343, 0.0750, 0.1058, 0.1336, 0.0580, 0.0614,
])


def points(n):
    rng = np.random.default_rng(2)
    q = np.zeros((n, 16), np.float32)
    q[:, 0:3] = rng.uniform((-6, 0.0, -6), (6, 0.5, 6), (64, 3))[:n]
    q[:, 3] = 1.0
    d = rng.normal(size=(64, 3))[:n]
    d[:, 1] = np.abs(d[:, 1])
    q[:, 4:7] = d / np.linalg.norm(d, axis=1, keepdims=True)
    q[:, 9] = 1.0
    return q


def test_frames_learn_what_the_arrival_order_gives():
    n, rays = 9000, 36
    ctx = bp.LuxContext()
    scene = bp.GpuScene(ctx, packed("atrium65536"))
    pos, nrm = floor_receivers(n, 21, extent=6.0)
    d_pos, d_nrm = to_device(pos), to_device(nrm)
    view = bp.SplitView(ctx, max_receivers=n, max_cells=1 << 16, max_entries=1 << 25, max_rays=n * rays)
    cache = bp.LearnedCache(ctx, batch=4096, seed=3)
    cache.set_bounds((-8, -1, -8), (8, 11, 8))
    view.set_cache(cache, cutoff_level=2, validate_period=4, error_bound=64.0, train_samples=65536, fallback_frames=4)
    for frame in range(2):
        settings = bp.RadianceCascades(frame_index=frame, probe_spacing=0.25, interval_length=0.4, levels=8,
                                       interval_ratio=2.0, rays_per_receiver=rays, emissive_samples=16).sanitized()
        view.trace_merge(scene, settings, d_pos.data_ptr(), d_nrm.data_ptr(), n)
    assert view.cache_stats().trained_samples == 65536
    query, out = to_device(points(len(PREDICTED))), empty_device(len(PREDICTED) * 16)
    cache.query(query.data_ptr(), len(PREDICTED), out.data_ptr())
    ctx.synchronize()
    got = from_device(out, np.float32, (len(PREDICTED), 4))[:, :3].mean(1)
    # Runs are within 4% of it; the mixture of another chain of loads is some 45% off.
    assert np.linalg.norm(got - PREDICTED) < 0.15 * np.linalg.norm(PREDICTED)
