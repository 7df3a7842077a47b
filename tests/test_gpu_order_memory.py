"""When a view orders its visibility queries without being asked, and the
memory it takes for that."""
import numpy as np
import pytest

import bevy_penumbra_b200 as bp
from tests.helpers import packed, to_device
from tests.test_gpu_batch import floor_receivers

pytestmark = pytest.mark.gpu

# Receivers of sixteen rays with eight samples each: 2^21 possible queries and
# the first count below; frames of 6 x 2^20 take the finer grid.
AT = 1 << 14
SETTINGS = dict(probe_spacing=0.25, interval_length=0.4, levels=4, rays_per_receiver=16, emissive_samples=16)


def free_bytes():
    import torch

    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


class Frames:
    def __init__(self, most, stream=None):
        self.ctx = bp.LuxContext(0, stream.cuda_stream) if stream else bp.LuxContext()
        self.scene = bp.GpuScene(self.ctx, packed("atrium65536"))
        pos, nrm = floor_receivers(most, 7, extent=6.0)
        self.pos, self.nrm = to_device(pos), to_device(nrm)
        self.view = bp.SplitView(self.ctx, max_receivers=most, max_cells=1 << 16, max_entries=1 << 24,
                                 max_rays=most * 16)
        self.settings = bp.RadianceCascades(**SETTINGS).sanitized()

    def run(self, count):
        self.view.trace_merge(self.scene, self.settings, self.pos.data_ptr(), self.nrm.data_ptr(), count)

    def hits(self, count):
        self.run(count)
        assert self.view.stats().error_flags == 0
        return self.view.read_hits(count * 16)


def test_room_for_the_order_is_made_once_for_the_largest_frame():
    f = Frames(4 * AT)
    f.run(AT - 1)
    before = free_bytes()
    f.run(AT - 1)
    assert free_bytes() == before
    f.run(AT)  # the first frame that is ordered
    ordered = free_bytes()
    assert before - ordered >= 68 * 4 * AT * 16 + (64 << 20)
    for count in (2 * AT, 3 * AT + 1, 4 * AT, AT):  # past 6 x 2^20 queries and back
        f.run(count)
    assert free_bytes() == ordered


def test_a_tuning_that_does_not_ask_orders_nothing():
    f = Frames(2 * AT)
    f.view.set_tuning(sort_queries=0)
    f.run(AT - 1)
    before = free_bytes()
    f.run(2 * AT)
    assert free_bytes() == before


def test_a_captured_frame_does_not_allocate():
    """A large frame under stream capture, in a view that has not ordered yet,
    runs in the order the queries come in; the same hits."""
    import torch

    stream = torch.cuda.Stream()
    f = Frames(2 * AT, stream)
    want = Frames(2 * AT).hits(2 * AT)
    f.run(64)  # streams and events exist from the first frame on
    f.ctx.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(stream):
        graph.capture_begin()
        f.run(2 * AT)
        graph.capture_end()
        graph.replay()
    stream.synchronize()
    got = f.view.read_hits(2 * AT * 16)
    for field in ("triangle", "instance", "errors"):
        np.testing.assert_array_equal(got[field], want[field], err_msg=field)
    np.testing.assert_array_equal(got["distance"].view(np.uint32), want["distance"].view(np.uint32))
