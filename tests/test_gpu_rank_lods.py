"""The sample-sequence order by cell ranks against the order by 62-bit keys in
frames with distance LODs, where a cell's LOD is part of its place."""
import numpy as np
import pytest

import bevy_penumbra_b200 as bp
from bevy_penumbra_b200 import scenes
from tests.helpers import packed, to_device

pytestmark = pytest.mark.gpu

RANKED = 1 << 17  # places for cells up to which they are ranked


def hits(pos, cells, keep):
    nrm = np.zeros_like(pos)
    nrm[:, 1] = 1.0
    settings = bp.RadianceCascades(levels=3, rays_per_receiver=1, frame_index=7).sanitized()
    ctx = bp.LuxContext()
    scene = bp.GpuScene(ctx, packed("atrium65536"))
    view = bp.SplitView(ctx, max_receivers=len(pos), max_cells=cells, max_entries=1 << 25, max_rays=len(pos))
    eye = (0.0, 1.5, 0.0)
    view.set_camera(scenes.clip_from_world(eye, (3.0, 1.0, 3.0), 60.0, 64, 64), eye, 64, 8)
    d_pos, d_nrm = to_device(pos), to_device(nrm)
    view.trace_merge(scene, settings, d_pos.data_ptr(), d_nrm.data_ptr(), len(pos))
    assert view.stats().error_flags == 0
    return view.read_hits(len(pos))[:keep]


# Receivers of many LODs; twice as many places with LODs as receivers.
@pytest.mark.parametrize("n", [65, 1025, 16384])
def test_ranks_and_full_keys_order_lods_the_same(n):
    rng = np.random.default_rng(n)
    pos = np.zeros((n, 4), np.float32)
    scale = np.exp(rng.uniform(np.log(0.5), np.log(60.0), n))
    pos[:, :3] = rng.uniform((-1.0, 0.0, -1.0), (1.0, 0.2, 1.0), (n, 3)) * scale[:, None]
    ranked = hits(pos, RANKED, n)
    far = np.zeros((RANKED // 2 + 1, 4), np.float32)
    far[:, :3] = 60000.0  # one far cell, after every other: 2 (n + these) places are too many to rank
    full = hits(np.concatenate([pos, far]), 2 * RANKED, n)
    for field in ("triangle", "instance", "errors"):
        np.testing.assert_array_equal(ranked[field], full[field], err_msg=field)
    np.testing.assert_array_equal(ranked["distance"].view(np.uint32), full["distance"].view(np.uint32))
