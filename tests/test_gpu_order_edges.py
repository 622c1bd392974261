"""Material-ordered shading at the edges of its tiles (512 queue positions) and of a warp: the image is the
queue-ordered one, bit for bit, for a single render and for the same image as a batched request."""
import pytest

import lambent_b200 as lb
from lambent_b200 import _abi, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,spp", [(1, 1, 1), (31, 1, 1), (511, 1, 1), (512, 1, 1), (513, 1, 1), (73, 71, 3), (512, 37, 2)])
def test_orders_agree(cuda, w, h, spp):
    import torch
    s = scenes.textured_cornell(w, h)
    g = lb.GpuScene(s)
    images = []
    for order in (_abi.SHADE_ORDER_QUEUE, _abi.SHADE_ORDER_MATERIAL):
        pipe = lb.RayTracer(lb.path_tracing.Medium).create_pipeline(*s.layout_counts(), lb.PathTracerOpts(
            samples=spp, restir_temporal=_abi.RESTIR_DISABLED, max_depth=6))
        pipe.set_shade_order(order)
        single, batched = (torch.full((h, w, 4), -1.0, device="cuda") for _ in range(2))
        bufs = lb.DataBuffers(w, h, 1, 0)
        for _ in range(2):  # the second render finds the first one's counters
            pipe.render(g, bufs, s.camera, lb.targets_from(single), 5)
        pipe.batch_render([(g, s.camera, lb.targets_from(batched), spp, 5)])
        torch.cuda.synchronize()
        assert pipe.stats().error_flags == 0
        images += [single, batched]
    assert (images[0][..., 3] == 1.0).all()
    for im in images[1:]:
        assert torch.equal(im.view(torch.int32), images[0].view(torch.int32))
