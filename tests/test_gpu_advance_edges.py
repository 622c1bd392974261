"""DataBuffers::advance_frame at the edges of its kernels' blocks (64 world cells; 256 16-byte words of
reservoirs and screen chains), against the oracle's end-of-frame passes."""
import ctypes

import numpy as np
import pytest

import lambent_b200 as lb
from lambent_b200 import _abi
from oracle import oracle_py as O

pytestmark = pytest.mark.gpu


def copy(dst, src, nbytes, kind):
    import torch
    torch.cuda.synchronize()
    rt = ctypes.CDLL("libcudart.so")
    assert rt.cudaMemcpy(ctypes.c_void_p(dst), ctypes.c_void_p(src), ctypes.c_size_t(nbytes), kind) == 0


def put(bufs, which, a):
    ptr, size = bufs.device_buffer(which)
    assert a.nbytes == size
    copy(ptr, a.ctypes.data, size, 1)


def get(bufs, which):
    ptr, size = bufs.device_buffer(which)
    a = np.empty(size, np.uint8)
    copy(a.ctypes.data, ptr, size, 2)
    return a.view(np.uint32)


@pytest.mark.parametrize("w,h,cells", [(1, 1, 1), (63, 1, 63), (64, 1, 64), (65, 1, 65), (37, 19, 1027)])
def test_advance(cuda, w, h, cells):
    rng = np.random.default_rng(cells)
    bufs = lb.DataBuffers(w, h, cells, _abi.BUFFER_ALL)
    res = rng.random((w * h, 16)).astype(np.float32)
    res.view(np.uint32)[:, 14] = rng.integers(0, 60, w * h).astype(np.uint32) | (rng.integers(0, 2, w * h).astype(np.uint32) << 31)
    chains = rng.random((w * h, 8)).astype(np.float32)
    world = rng.random((cells, 14)).astype(np.float32)
    u = world.view(np.uint32)
    u[:, 1] = rng.integers(0, 20, cells)
    u[:, 5] = rng.integers(0, 2, cells)
    u[:, 13] = rng.integers(0, 4, cells)
    put(bufs, lb.DataBuffers.RESERVOIRS, res)
    put(bufs, lb.DataBuffers.CHAINS, chains)
    put(bufs, lb.DataBuffers.WORLD, world)
    bufs.advance_frame(_abi.BUFFER_ALL, lb.AdvanceOptions(20))
    want_res, want_world = res.copy(), world.view(np.uint32).reshape(-1).copy()
    O.process_gi(want_res, 20)
    O.process_world(want_world)
    np.testing.assert_array_equal(get(bufs, lb.DataBuffers.OLD_RESERVOIRS), want_res.view(np.uint32).reshape(-1))
    np.testing.assert_array_equal(get(bufs, lb.DataBuffers.OLD_CHAINS), chains.view(np.uint32).reshape(-1))
    np.testing.assert_array_equal(get(bufs, lb.DataBuffers.WORLD), want_world)
    np.testing.assert_array_equal(get(bufs, lb.DataBuffers.OLD_WORLD), want_world)
    assert not get(bufs, lb.DataBuffers.RESERVOIRS).any() and not get(bufs, lb.DataBuffers.CHAINS).any()
