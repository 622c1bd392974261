"""Data buffers whose resize failed: the passes over them are refused, and a resize that succeeds makes them
whole again.  (More pixels than any device holds: the allocation fails at once.)"""
import pytest

import lambent_b200 as lb
from lambent_b200 import _abi, scenes

pytestmark = pytest.mark.gpu


def test_passes_after_a_resize_that_failed(cuda):
    import torch
    s = scenes.cornell_box(48, 32)
    g = lb.GpuScene(s)
    pipe = lb.RayTracer(lb.path_tracing.Medium).create_pipeline(*s.layout_counts(), lb.PathTracerOpts(
        samples=1, restir_temporal=_abi.RESTIR_PER_PIXEL))

    def frame(bufs):
        col, out = (torch.zeros((32, 48, 4), device="cuda") for _ in range(2))
        pipe.render(g, bufs, s.camera, lb.targets_from(col), 5)
        bufs.temporal_resampling(5)
        bufs.spatial_resampling(lb.targets_from(out), 3, 31, 5)
        bufs.advance_frame(_abi.BUFFER_ALL, lb.AdvanceOptions(20))
        torch.cuda.synchronize()
        return torch.stack([col, out])

    want = frame(lb.DataBuffers(48, 32, 64, _abi.BUFFER_ALL))
    bufs = lb.DataBuffers(48, 32, 64, _abi.BUFFER_ALL)
    with pytest.raises(lb.LambentError):
        bufs.resize(65535, 65535)
    for call in (lambda: frame(bufs), lambda: bufs.advance_frame(_abi.BUFFER_ALL, lb.AdvanceOptions(20)), lambda: bufs.temporal_resampling(5),
                 lambda: bufs.spatial_resampling(lb.targets_from(torch.zeros((32, 48, 4), device="cuda")), 3, 31, 5)):
        with pytest.raises(lb.LambentError) as e:
            call()
        assert e.value.code == _abi.ERR_INVALID_ARGUMENT
    bufs.resize(48, 32)
    assert torch.equal(frame(bufs), want)
