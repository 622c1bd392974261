"""Device memory of a render's wave: what the renders of each kind take for a path, and waves of sizes at
which an estimate could go wrong."""
import pytest

import lambent_b200 as lb
from lambent_b200 import _abi, scenes

pytestmark = pytest.mark.gpu


def _render(torch, s, w, h, spp, guide_mode=_abi.GUIDE_NONE, restir=_abi.RESTIR_DISABLED, wave_paths=0):
    pipe = lb.RayTracer(lb.path_tracing.Medium).create_pipeline(*s.layout_counts(), lb.PathTracerOpts(
        samples=spp, restir_temporal=restir, max_depth=2, guide_mode=guide_mode))
    guide = None
    if guide_mode & _abi.GUIDE_LEARNED:
        guide = lb.Guide(lb.GuideOptions(record_capacity=0, train_spp=0))
        pipe.set_guide(guide)
    pipe.set_wave_paths(wave_paths)
    g, bufs = lb.GpuScene(s), lb.DataBuffers(w, h, 1 << 10, _abi.BUFFER_ALL)
    col = torch.zeros((h, w, 4), device="cuda")
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    pipe.render(g, bufs, s.camera, lb.targets_from(col), 3)
    torch.cuda.synchronize()
    return col, before - torch.cuda.mem_get_info()[0]


@pytest.mark.parametrize("mode,restir,per_path", [
    (_abi.GUIDE_NONE, _abi.RESTIR_DISABLED, 200), (_abi.GUIDE_NONE, _abi.RESTIR_PER_PIXEL, 296),
    (_abi.GUIDE_LEARNED, _abi.RESTIR_DISABLED, 352)], ids=["plain", "restir", "learned"])
def test_bytes_per_path(cuda, mode, restir, per_path):
    """The wave takes what its layout says: the arrays of 4M paths and of their pixels, and no more than
    the driver's rounding and the first launches' own memory besides."""
    import torch
    s = scenes.cornell_box(512, 512)
    _render(torch, s, 16, 16, 2, mode, restir)  # the kernels' modules and local memory
    _, used = _render(torch, s, 512, 512, 16, mode, restir)
    arrays = per_path * 512 * 512 * 16
    assert arrays <= used <= arrays + 64 * 512 * 512 + (64 << 20)


@pytest.mark.parametrize("w,h", [(1, 1), (1, 63), (64, 1)])
@pytest.mark.parametrize("wave_paths", [0, 1, 100])
def test_tiny_images(cuda, w, h, wave_paths):
    import torch
    s = scenes.cornell_box(w, h)
    whole, _ = _render(torch, s, w, h, 7)
    part, _ = _render(torch, s, w, h, 7, wave_paths=wave_paths)
    assert torch.equal(whole, part)
