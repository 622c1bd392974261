"""The shared triangle phase with more triangles than its list holds (256): a node whose 24 triangles all lie
in one box, and warps full of equal rays, so that each of up to 32 lanes exposes all 24 at once and the
phase takes up to three rounds.  Closest hits against the CPU oracle; an any-hit ray's answer against the
closest hits and against the ray on its own, whose 24 triangles fit the list."""
import numpy as np
import pytest

import lambent_b200 as lb
from lambent_b200 import _abi, scenes
from oracle import oracle_py as O
from test_gpu_trace_queues import gpu_trace, same

pytestmark = pytest.mark.gpu

LIST, SMALL_WARPS = 256, 8  # COOP_LIST, and the warps per SM that a small queue is spread over


def one_node(flags):
    s = scenes.textured_cornell(16, 16)
    rng = np.random.default_rng(3)
    tris = []
    for k in range(24):  # equal boxes, different planes: the builder can only halve them, down to leaves of 3
        z, m = (-1.0 if k & 1 else 1.0), rng.uniform(-0.9, 0.9)
        tris += [(-1.0, -1.0, z), (1.0, -1.0, -z), (m if k & 2 else -m, 1.0, m)]
    s.blas[0].update(vertices=np.asarray(tris, np.float32), indices=None, flags=flags)
    s.instances[0]["material_indices"] = np.arange(24, dtype=np.uint32) % 5
    if not flags:
        for tex in s.diffuse:
            tex[rng.random(tex.shape[:2]) < 0.4, 3] = 0
    return s


@pytest.mark.parametrize("flags", [1, 0], ids=["opaque", "alpha_tested"])
def test_more_triangles_than_the_list_holds(cuda, flags):
    import torch
    s = one_node(flags)
    g = lb.GpuScene(s)
    assert g.stats().triangle_count == 24 and g.stats().blas_node_count == 1
    n = 64 * 1024
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert n >= 32 * SMALL_WARPS * sms and 26 * 24 > LIST  # a warp holds 26 to 32 rays
    rng = np.random.default_rng(5)
    one = np.zeros((n // 64, 8), np.float32)
    one[:, 0:2] = rng.uniform(-0.6, 0.6, (n // 64, 2))
    one[:, 2] = 3.0
    one[:, 4:6] = rng.uniform(-0.1, 0.1, (n // 64, 2))
    one[:, 6] = -1.0
    one[:, 3], one[:, 7] = 1e-4, 1000.0
    rays = np.repeat(one, 64, axis=0)
    want = np.repeat(O.OracleScene(s).trace(one, bruteforce=True), 64)
    assert (want["kind"] != 0).mean() > 0.8
    closest = gpu_trace(g, rays)
    same(closest, want)
    anyh = gpu_trace(g, rays, _abi.TRACE_ANY)
    np.testing.assert_array_equal(anyh["kind"] != 0, closest["kind"] != 0)
    hit = anyh["kind"] != 0
    assert (anyh["t"][hit] >= closest["t"][hit]).all()
    same(anyh, np.repeat(anyh[::64], 64))  # all rays of a bundle alike
    for k in range(0, n, n // 16):
        same(gpu_trace(g, rays[k:k + 1], _abi.TRACE_ANY), anyh[k:k + 1])
