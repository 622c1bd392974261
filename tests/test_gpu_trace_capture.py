"""A ray query waits for its stream, so it fails in a stream capture; the calls after it run as before."""
import pytest

import lambent_b200 as lb
from lambent_b200 import _abi, scenes

pytestmark = pytest.mark.gpu


def captured_query(g, rays, hits, side):
    from cuda.bindings import driver
    err, = driver.cuStreamBeginCapture(side.cuda_stream, driver.CUstreamCaptureMode.CU_STREAM_CAPTURE_MODE_THREAD_LOCAL)
    assert err == driver.CUresult.CUDA_SUCCESS
    with pytest.raises(lb.LambentError):
        g.trace(rays, hits, stream=side)
    err, _ = driver.cuStreamEndCapture(side.cuda_stream)
    assert err == driver.CUresult.CUDA_ERROR_STREAM_CAPTURE_INVALIDATED


def box_and_rays(torch):
    s = scenes.cornell_box(16, 16)
    rays = torch.zeros((256, 8), device="cuda")
    rays[:, 1], rays[:, 2], rays[:, 6], rays[:, 7] = 1.0, 3.0, -1.0, 1000.0
    return s, lb.GpuScene(s), rays


def test_an_error_that_was_returned_is_not_the_next_calls(cuda):
    """Neither the next render, which looks at the runtime's last error, nor the program's own calls."""
    import torch
    s, g, rays = box_and_rays(torch)
    hits = torch.full((256, 6), -1, dtype=torch.int32, device="cuda")
    col = torch.zeros((16, 16, 4), device="cuda")
    pipe = lb.RayTracer(lb.path_tracing.Medium).create_pipeline(*s.layout_counts(), lb.PathTracerOpts(
        samples=1, restir_temporal=_abi.RESTIR_DISABLED))
    torch.cuda.synchronize()
    captured_query(g, rays, hits, torch.cuda.Stream())
    pipe.render(g, lb.DataBuffers(16, 16, 1, 0), s.camera, lb.targets_from(col), 0)
    torch.cuda.synchronize()
    captured_query(g, rays, hits, torch.cuda.Stream())
    assert (hits == -1).all()  # captured, not run


def test_queries_refused_in_a_capture_keep_no_slot(cuda):
    """With its 64 scratch slots taken, a scene's queries allocate from the device's memory pool."""
    import torch
    from cuda.bindings import driver
    _, g, rays = box_and_rays(torch)
    want, got = (torch.full((256, 6), -1, dtype=torch.int32, device="cuda") for _ in range(2))
    g.trace(rays, want)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    for _ in range(70):
        captured_query(g, rays, got, side)
    torch.cuda.synchronize()
    assert (got == -1).all()
    err, pool = driver.cuDeviceGetDefaultMemPool(0)
    assert err == driver.CUresult.CUDA_SUCCESS
    attr = driver.CUmemPool_attribute.CU_MEMPOOL_ATTR_USED_MEM_HIGH
    driver.cuMemPoolSetAttribute(pool, attr, driver.cuuint64_t(0))
    for _ in range(4):
        got.fill_(-1)
        g.trace(rays, got)
        torch.cuda.synchronize()
        assert torch.equal(got, want)
    err, high = driver.cuMemPoolGetAttribute(pool, attr)
    assert err == driver.CUresult.CUDA_SUCCESS and int(high) == 0
