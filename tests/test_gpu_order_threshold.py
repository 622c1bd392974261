"""The automatic shading order on both sides of its threshold (2^18 paths in a wave): which order ran shows
in the number of launches, one more per bounce in material order; the images are those of either."""
import pytest

import lambent_b200 as lb
from lambent_b200 import _abi, scenes

pytestmark = pytest.mark.gpu

AUTO, QUEUE, MATERIAL = _abi.SHADE_ORDER_AUTO, _abi.SHADE_ORDER_QUEUE, _abi.SHADE_ORDER_MATERIAL
DEPTH = 4


def _pipe(s, spp, order):
    pipe = lb.RayTracer(lb.path_tracing.Medium).create_pipeline(*s.layout_counts(), lb.PathTracerOpts(
        samples=spp, restir_temporal=_abi.RESTIR_DISABLED, max_depth=DEPTH))
    pipe.set_shade_order(order)
    return pipe


SIZES = [(511, 513, 1, False), (512, 512, 1, True), (513, 512, 1, True), (257, 255, 4, False), (256, 256, 4, True)]


@pytest.mark.parametrize("w,h,spp,sorts", SIZES)
def test_single_render(cuda, w, h, spp, sorts):
    import torch
    s = scenes.textured_cornell(w, h)
    g = lb.GpuScene(s)
    images, launches = {}, {}
    for order in (AUTO, QUEUE, MATERIAL):
        pipe = _pipe(s, spp, order)
        images[order] = torch.full((h, w, 4), -1.0, device="cuda")
        pipe.render(g, lb.DataBuffers(w, h, 1, 0), s.camera, lb.targets_from(images[order]), 5)
        torch.cuda.synchronize()
        launches[order] = pipe.stats().kernel_launches
    assert launches[MATERIAL] == launches[QUEUE] + DEPTH
    assert launches[AUTO] == launches[MATERIAL if sorts else QUEUE]
    assert torch.equal(images[AUTO], images[QUEUE]) and torch.equal(images[AUTO], images[MATERIAL])


@pytest.mark.parametrize("graph", [0, 1])
@pytest.mark.parametrize("w,h,spp,sorts", SIZES[:3])
def test_batch(cuda, w, h, spp, sorts, graph):
    """Two requests that fill one wave to just below, at and above the threshold; the order changed on
    one pipeline between the calls, so that a captured graph is rebuilt."""
    import torch
    s = scenes.textured_cornell(w, h)
    g = lb.GpuScene(s)
    pipe = _pipe(s, spp, AUTO)
    rows = h // 2
    images, launches = {}, {}
    for order in (AUTO, QUEUE, MATERIAL, AUTO):
        pipe.set_shade_order(order)
        out = [torch.full((r, w, 4), -1.0, device="cuda") for r in (rows, h - rows)]
        pipe.batch_render([(g, s.camera, lb.targets_from(o), spp, 5 + k) for k, o in enumerate(out)],
                          _abi.BatchTuning(use_graph=graph))
        torch.cuda.synchronize()
        assert pipe.stats().error_flags == 0
        n = pipe.stats().kernel_launches
        images.setdefault(order, out)
        assert n == launches.setdefault(order, n)
        for a, b in zip(out, images[AUTO]):
            assert torch.equal(a, b)
    assert launches[MATERIAL] == launches[QUEUE] + DEPTH
    assert launches[AUTO] == launches[MATERIAL if sorts else QUEUE]


def test_graph_is_rebuilt_when_the_order_changes(cuda):
    """Small requests, whose automatic order is the queue's: material order, queue order and back, each
    with the images of the requests rendered alone."""
    import torch
    specs = [(scenes.cornell_box(64, 48), 5, 11), (scenes.textured_cornell(80, 80), 9, 33),
             (scenes.textured_cornell(128, 96), 4, 55)]
    gpu = [lb.GpuScene(s) for s, _, _ in specs]
    alone = []
    for (s, spp, seed), g in zip(specs, gpu):
        col = torch.zeros((s.height, s.width, 4), device="cuda")
        _pipe(s, spp, QUEUE).render(g, lb.DataBuffers(s.width, s.height, 1, 0), s.camera, lb.targets_from(col), seed)
        alone.append(col)
    pipe = lb.RayTracer(lb.path_tracing.Medium).create_pipeline(8, 8, 8, 8, lb.PathTracerOpts(
        samples=1, restir_temporal=_abi.RESTIR_DISABLED, max_depth=DEPTH))
    out = [torch.zeros_like(c) for c in alone]
    requests = [(g, s.camera, lb.targets_from(o), spp, seed) for (s, spp, seed), g, o in zip(specs, gpu, out)]
    captured = []
    for order in (MATERIAL, MATERIAL, QUEUE, MATERIAL):
        pipe.set_shade_order(order)
        for o in out:
            o.zero_()
        pipe.batch_render(requests, _abi.BatchTuning(wave_paths=32 * 1024, use_graph=1))
        torch.cuda.synchronize()
        captured.append(pipe.stats().kernel_launches)
        for o, c in zip(out, alone):
            assert torch.equal(o, c)
    assert captured[0] == captured[3] > captured[2] > 0  # each change of order captures the batch again
