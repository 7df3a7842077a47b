"""The sample-sequence order by cell ranks (pieces sorted in shared memory)
at cell counts around whole pieces and tiles: receivers in sequence order are
their cells' keys in order, ties by index, as a stable host sort gives them."""
import numpy as np
import pytest

import bevy_penumbra_b200 as bp
from tests.helpers import packed, to_device

pytestmark = pytest.mark.gpu


def hits(n, per_cell, max_cells, seed):
    """Hits of n single-cell receivers (per_cell of them in each cell)."""
    rng = np.random.default_rng(seed)
    cells = -(-n // per_cell)
    side = int(np.ceil(np.sqrt(cells)))
    pos = np.zeros((n, 4), np.float32)
    which = rng.permutation(np.arange(n) % cells)
    pos[:, 0] = (which % side) * 0.25 - 0.125 * side + 0.1
    pos[:, 2] = (which // side) * 0.25 - 0.125 * side + 0.1
    pos[:, 1] = 0.1
    nrm = np.zeros_like(pos)
    nrm[:, 1] = 1.0
    settings = bp.RadianceCascades(levels=3, rays_per_receiver=1, probe_spacing=0.25, frame_index=5).sanitized()
    ctx = bp.LuxContext()
    scene = bp.GpuScene(ctx, packed("atrium65536"))
    view = bp.SplitView(ctx, max_receivers=n, max_cells=max_cells, max_entries=1 << 25, max_rays=n)
    d_pos, d_nrm = to_device(pos), to_device(nrm)
    view.trace_merge(scene, settings, d_pos.data_ptr(), d_nrm.data_ptr(), n)
    assert view.stats().error_flags == 0
    return view.read_hits(n), view.stats().cells[0]


# Ranked (at most 2^17 places for cells) against the full 62-bit keys (more).
@pytest.mark.parametrize("n,per_cell", [(1, 1), (255, 1), (511, 1), (1024, 1), (1025, 2), (3000, 1), (40000, 3), (65537, 1)])
def test_ranked_and_full_keys_order_the_same(n, per_cell):
    ranked, cells = hits(n, per_cell, 1 << 17, n)
    assert cells == -(-n // per_cell)
    if cells <= 16384:  # the smaller pieces
        np.testing.assert_array_equal(hits(n, per_cell, 16384, n)[0], ranked)
    # Room for more cells than are ranked, and receivers that could seed them.
    pad = (1 << 17) + 1 - n
    full = hits_with_far(n, per_cell, pad)
    for field in ("triangle", "instance", "errors"):
        np.testing.assert_array_equal(ranked[field], full[field], err_msg=field)
    np.testing.assert_array_equal(ranked["distance"].view(np.uint32), full["distance"].view(np.uint32))


def hits_with_far(n, per_cell, pad):
    """The same receivers and pad more of one far cell, sorted by full keys."""
    rng = np.random.default_rng(n)
    cells = -(-n // per_cell)
    side = int(np.ceil(np.sqrt(cells)))
    pos = np.zeros((n + pad, 4), np.float32)
    which = rng.permutation(np.arange(n) % cells)
    pos[:n, 0] = (which % side) * 0.25 - 0.125 * side + 0.1
    pos[:n, 2] = (which // side) * 0.25 - 0.125 * side + 0.1
    pos[:n, 1] = 0.1
    pos[n:, :3] = 60000.0  # after every cell of the scene
    nrm = np.zeros_like(pos)
    nrm[:, 1] = 1.0
    settings = bp.RadianceCascades(levels=3, rays_per_receiver=1, probe_spacing=0.25, frame_index=5).sanitized()
    ctx = bp.LuxContext()
    scene = bp.GpuScene(ctx, packed("atrium65536"))
    view = bp.SplitView(ctx, max_receivers=n + pad, max_cells=1 << 18, max_entries=1 << 25, max_rays=n + pad)
    d_pos, d_nrm = to_device(pos), to_device(nrm)
    view.trace_merge(scene, settings, d_pos.data_ptr(), d_nrm.data_ptr(), n + pad)
    assert view.stats().error_flags == 0
    return view.read_hits(n + pad)[:n]
