"""What a pipeline keeps from one lam_batch_render to the next: the captured graph and the request
tables."""
import ctypes as C

import pytest

import lambent_b200 as lb
from lambent_b200 import _abi, scenes

pytestmark = pytest.mark.gpu


def _pipe(samples=2, depth=5):
    opts = lb.PathTracerOpts(samples=samples, restir_temporal=_abi.RESTIR_DISABLED, max_depth=depth)
    return lb.RayTracer(lb.path_tracing.Medium).create_pipeline(8, 8, 8, 8, opts)


def _single(g, s, spp, seed):
    import torch
    col = torch.zeros((s.height, s.width, 4), device="cuda")
    _pipe(spp).render(g, lb.DataBuffers(s.width, s.height, 1, 0), s.camera, lb.targets_from(col), seed)
    torch.cuda.synchronize()
    return col


def _cutout():
    s = scenes.textured_cornell(64, 48)
    s.blas[0]["flags"] = 0
    for tex in s.diffuse:
        tex[::2, :, 3] = 0
    return s


def test_graph_of_opaque_scenes_is_not_replayed_for_a_cutout_at_the_same_address(cuda):
    """The captured graph holds the traversal kernel for opaque geometry; a new scene is usually
    created where a destroyed one of the same size was."""
    import torch
    opaque, cutout = scenes.textured_cornell(64, 48), _cutout()
    pipe = _pipe()
    col = torch.zeros((48, 64, 4), device="cuda")
    tuning = _abi.BatchTuning(use_graph=1)

    def render(g):
        pipe.batch_render([(g, opaque.camera, lb.targets_from(col), 2, 3)], tuning)
        torch.cuda.synchronize()
        return col.clone()

    g = lb.GpuScene(opaque)
    address = g._h.value
    first = render(g)
    assert torch.equal(first, _single(g, opaque, 2, 3))
    # Empty the allocator's list of free blocks of this size, so that the scene's block comes to its head,
    # and put blocks before it for what lam_scene_create allocates besides the scene.
    libc = C.CDLL(None)
    libc.malloc.restype = C.c_void_p
    libc.malloc.argtypes = libc.malloc_usable_size.argtypes = [C.c_size_t]
    libc.free.argtypes = [C.c_void_p]
    size = libc.malloc_usable_size(address)
    blocks = [libc.malloc(size) for _ in range(256)]
    pipe._batch_keep = None  # a C-ABI caller's batch holds no scene
    del g
    for b in blocks[:5]:
        libc.free(b)
    cutouts = [lb.GpuScene(cutout)]
    while cutouts[-1]._h.value != address and len(cutouts) < 64:
        cutouts.append(lb.GpuScene(cutout))
    for b in blocks[5:]:
        libc.free(b)
    assert cutouts[-1]._h.value == address, "no scene was created where the destroyed one was"
    second = render(cutouts[-1])
    assert torch.equal(second, _single(cutouts[-1], cutout, 2, 3))
    assert not torch.equal(first, second)


@pytest.mark.parametrize("graph", [0, 1])
def test_batches_issued_back_to_back(cuda, graph):
    """Different requests with no wait between the calls: a batch's tables stay as they are until it
    has run."""
    import torch
    s = [scenes.cornell_box(160, 120), scenes.textured_cornell(64, 48), scenes.occluded_cornell(33, 47)]
    g = [lb.GpuScene(x) for x in s]
    batches = [[(0, 16, 1), (1, 7, 2)], [(2, 3, 3)], [(1, 5, 4), (2, 2, 5), (0, 1, 6), (1, 1, 7)]] * 2
    cols = [[torch.full((s[k].height, s[k].width, 4), -1.0, device="cuda") for k, _, _ in b] for b in batches]
    pipe = _pipe()
    torch.cuda.synchronize()
    for b, out in zip(batches, cols):
        pipe.batch_render([(g[k], s[k].camera, lb.targets_from(o), spp, seed) for (k, spp, seed), o in zip(b, out)],
                          _abi.BatchTuning(wave_paths=64 * 1024, use_graph=graph))
    torch.cuda.synchronize()
    assert pipe.stats().error_flags == 0
    for b, out in zip(batches, cols):
        for (k, spp, seed), o in zip(b, out):
            assert torch.equal(o, _single(g[k], s[k], spp, seed))
