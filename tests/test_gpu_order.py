"""The sample-sequence order by ranked cascade-0 cells (views whose receivers
seed few cells) against the order by full keys: the same rays, hence the same
hits, bit for bit."""
import numpy as np
import pytest

import bevy_penumbra_b200 as bp
from bevy_penumbra_b200 import scenes
from tests.helpers import packed, to_device

pytestmark = pytest.mark.gpu


def hits(scene, ctx, pos, nrm, max_cells, camera, frame):
    settings = bp.RadianceCascades(levels=4, rays_per_receiver=3, frame_index=frame).sanitized()
    view = bp.SplitView(ctx, max_receivers=len(pos), max_cells=max_cells, max_entries=1 << 24,
                        max_rays=len(pos) * settings.rays_per_receiver)
    if camera:
        eye = (0.0, 1.5, 0.0)
        view.set_camera(scenes.clip_from_world(eye, (3.0, 1.0, 3.0), 60.0, 64, 64), eye, 64, 8)
    d_pos, d_nrm = to_device(pos), to_device(nrm)
    view.trace_merge(scene, settings, d_pos.data_ptr(), d_nrm.data_ptr(), len(pos))
    assert view.stats().error_flags == 0
    return view.read_hits(len(pos) * settings.rays_per_receiver)


@pytest.mark.parametrize("n,camera", [(1, False), (33, False), (1025, True), (2049, False), (16383, True)])
def test_ranked_order_gives_the_rays_of_the_full_keys(n, camera):
    rng = np.random.default_rng(n)
    pos = np.zeros((n, 4), np.float32)
    pos[:, :3] = rng.uniform((-7.0, 0.0, -7.0), (7.0, 3.0, 7.0), (n, 3))
    pos[n // 2:, :3] = pos[:n - n // 2, :3] + np.float32(1e-3)  # many receivers per cell, far apart in index
    nrm = np.zeros_like(pos)
    nrm[:, 1] = 1.0
    ctx = bp.LuxContext()
    scene = bp.GpuScene(ctx, packed("atrium65536"))
    # Room for more cells than are ranked only where the receivers can seed
    # them; 16383 receivers with LODs can, so that frame sorts full keys
    # unless the view's capacity keeps it below.
    few, many = hits(scene, ctx, pos, nrm, 16384, camera, 7), None
    pad = 40000  # receivers that could seed more cells than are ranked, all in one far cell
    far = np.zeros((pad, 4), np.float32)
    far[:, :3] = (60000.0, 60000.0, 60000.0)  # sorts after every cell of the scene
    far_n = np.zeros_like(far)
    far_n[:, 1] = 1.0
    many = hits(scene, ctx, np.concatenate([pos, far]), np.concatenate([nrm, far_n]), 1 << 17, camera, 7)[:3 * n]
    for field in ("triangle", "instance", "errors"):
        np.testing.assert_array_equal(few[field], many[field], err_msg=field)
    np.testing.assert_array_equal(few["distance"].view(np.uint32), many["distance"].view(np.uint32))
