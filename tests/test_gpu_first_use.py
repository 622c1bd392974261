"""The first call on new objects in a non-blocking stream while the default stream is busy: what the calls
clear is cleared before their kernels run, not when the default stream gets to it."""
import pytest

import lambent_b200 as lb
from lambent_b200 import _abi, scenes

pytestmark = pytest.mark.gpu

BUSY = 100_000_000  # cycles of the default stream, 50 ms


def test_first_render_and_batch_beside_a_busy_default_stream(cuda):
    import torch
    s = scenes.textured_cornell(160, 96)
    g = lb.GpuScene(s)
    side = torch.cuda.Stream()

    def run(busy):
        a, out, b = (torch.zeros((96, 160, 4), device="cuda") for _ in range(3))
        torch.cuda.synchronize()
        if busy:
            torch.cuda._sleep(BUSY)
        bufs = lb.DataBuffers(160, 96, 64, _abi.BUFFER_ALL)
        frame = lb.RayTracer(lb.path_tracing.Medium).create_pipeline(*s.layout_counts(), lb.PathTracerOpts(
            samples=1, restir_temporal=_abi.RESTIR_PER_PIXEL))
        plain = lb.RayTracer(lb.path_tracing.Medium).create_pipeline(*s.layout_counts(), lb.PathTracerOpts(
            samples=1, restir_temporal=_abi.RESTIR_DISABLED))
        if busy:
            torch.cuda._sleep(BUSY)
        frame.render(g, bufs, s.camera, lb.targets_from(a), 5, stream=side)
        bufs.spatial_resampling(lb.targets_from(out), 3, 31, 5, stream=side)
        plain.batch_render([(g, s.camera, lb.targets_from(b), 3, 9)], stream=side)
        torch.cuda.synchronize()
        assert frame.stats().error_flags == plain.stats().error_flags == 0
        segments = frame.stats().ray_segments, plain.stats().ray_segments
        return torch.stack([a, out, b]), segments

    quiet, n = run(False)
    assert (quiet[..., 3] == 1.0).any() and min(n) > 0
    for _ in range(3):
        images, m = run(True)
        assert torch.equal(images, quiet) and m == n
