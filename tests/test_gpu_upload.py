"""A scene upload beside frames that are queued on the context's stream."""
import numpy as np
import pytest

import bevy_penumbra_b200 as bp
from tests.helpers import EMPTY, packed, to_device
from tests.test_gpu_radiance import random_rays

pytestmark = pytest.mark.gpu


def test_an_upload_does_not_wait_for_queued_work():
    import torch

    stream = torch.cuda.Stream()
    ctx = bp.LuxContext(0, stream.cuda_stream)
    first = bp.GpuScene(ctx, packed("atrium65536"))
    rays = random_rays(2000, (-7.0, 0.1, -7.0), (7.0, 4.0, 7.0), seed=2)
    d_rays = to_device(rays)
    out = [torch.zeros((len(rays), 8), dtype=torch.int32, device="cuda") for _ in range(2)]
    bp.trace_rays(ctx, first, d_rays.data_ptr(), len(rays), out[0].data_ptr())
    queued = torch.cuda.Event()
    torch.cuda.synchronize()
    with torch.cuda.stream(stream):
        torch.cuda._sleep(400_000_000)  # some 0.2 s of the stream
        queued.record()
    scene = bp.GpuScene(ctx, packed("atrium65536"))
    assert not queued.query()
    bp.trace_rays(ctx, scene, d_rays.data_ptr(), len(rays), out[1].data_ptr())
    stream.synchronize()
    near = [o.cpu().numpy() for o in out]
    assert np.mean(near[0][:, 1].view(np.uint32) != EMPTY) > 0.5
    np.testing.assert_array_equal(near[0], near[1])
