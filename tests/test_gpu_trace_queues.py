"""The traversal's queue and list edges: queues too small to fill the grid (spread over its warps), just
full and ragged; warps whose lanes expose more triangles in one step than the shared list holds; and
alpha-tested triangles in the shared phase.  Against the CPU oracle, or for any-hit queries, whose
triangle depends on the traversal order, against the closest hits and each ray on its own."""
import numpy as np
import pytest

import lambent_b200 as lb
from lambent_b200 import _abi, scenes
from oracle import oracle_py as O

pytestmark = pytest.mark.gpu


def gpu_trace(g, rays, mode=_abi.TRACE_CLOSEST):
    import torch
    r = torch.from_numpy(np.ascontiguousarray(rays, np.float32)).cuda()
    h = torch.full((rays.shape[0], 6), -1, dtype=torch.int32, device="cuda")
    g.trace(r, h, mode)
    torch.cuda.synchronize()
    return h.cpu().numpy().view(O.HIT_DTYPE).reshape(-1)


def same(a, b):
    for f in ("prim", "inst", "kind"):
        np.testing.assert_array_equal(a[f], b[f])
    for f in ("t", "u", "v"):
        np.testing.assert_allclose(a[f], b[f], rtol=3e-7, atol=0)  # 2 ulp


def box_rays(n, seed):
    rng = np.random.default_rng(seed)
    r = np.zeros((n, 8), np.float32)
    r[:, 0:3] = rng.uniform(-0.95, 0.95, (n, 3)) + np.array([0, 1, 0])
    r[:, 4:7] = rng.normal(size=(n, 3))
    r[:, 3], r[:, 7] = 1e-4, 1000.0
    return r


def cutout():
    s = scenes.cornell_box(16, 16)
    s.blas[0]["flags"] = 0
    tex = np.full((64, 64, 4), 200, np.uint8)
    tex[::2, :, 3] = 0
    s.diffuse = [tex.copy() for _ in s.diffuse]
    return s


@pytest.mark.parametrize("n", [1, 7, 8, 9, 31, 32, 33, 1000, 37889, 151553])
@pytest.mark.parametrize("make", [lambda: scenes.cornell_box(16, 16), cutout], ids=["opaque", "cutout"])
def test_queue_sizes(cuda, make, n):
    s = make()
    g = lb.GpuScene(s)
    rays = box_rays(n, n)
    closest = gpu_trace(g, rays)
    same(closest, O.OracleScene(s).trace(rays, bruteforce=True))
    anyh = gpu_trace(g, rays, _abi.TRACE_ANY)
    np.testing.assert_array_equal(anyh["kind"] != 0, closest["kind"] != 0)
    hit = anyh["kind"] != 0
    assert (anyh["t"][hit] >= closest["t"][hit]).all()
    for k in range(0, n, max(1, n // 8)):  # a ray's answer does not depend on the rays beside it
        same(gpu_trace(g, rays[k:k + 1], _abi.TRACE_ANY), anyh[k:k + 1])


@pytest.mark.parametrize("flags", [1, 0], ids=["opaque", "alpha_tested"])
def test_more_triangles_in_a_step_than_the_list_holds(cuda, flags):
    s = scenes.icosphere_field(64, 64, instances=3, subdiv=2, tex_size=16, tex_layers=2, seed=4)
    for b in s.blas:
        b["flags"] = flags
    g = lb.GpuScene(s)
    rng = np.random.default_rng(1)
    # bundles of 64 equal rays through an instance's centre: every lane of a warp exposes the same leaves
    rays = np.zeros((64 * 64, 8), np.float32)
    centre = np.stack([i["transform"].reshape(3, 4)[:, 3] for i in s.instances])[rng.integers(0, 3, 64)]
    d = rng.normal(size=(64, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    rays[:, 0:3] = np.repeat(centre - 6.0 * d, 64, axis=0)
    rays[:, 4:7] = np.repeat(d, 64, axis=0)
    rays[:, 3], rays[:, 7] = 1e-4, 1000.0
    o = O.OracleScene(s).trace(rays, bruteforce=True)
    assert (o["kind"] != 0).all()
    same(gpu_trace(g, rays), o)
