"""A view gives back what it took."""
import pytest

import bevy_penumbra_b200 as bp

pytestmark = pytest.mark.gpu


def test_destroyed_views_leave_no_device_memory_behind():
    import torch

    ctx = bp.LuxContext()

    def free_after(views):
        for _ in range(views):
            bp.SplitView(ctx, max_receivers=256, max_cells=1 << 10, max_entries=1 << 24, max_rays=256).close()
        torch.cuda.synchronize()
        return torch.cuda.mem_get_info()[0]

    before = free_after(2)
    assert free_after(8) == before
