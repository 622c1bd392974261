"""Ray queries in flight at once: each has its own work counter and error flags, from the scene's 64
slots or, with all of those taken, from an allocation of its own."""
import threading

import pytest

import lambent_b200 as lb
from lambent_b200 import scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("threads", [2, 64, 80])
def test_queries_of_many_threads_and_streams(cuda, threads):
    import torch
    g = lb.GpuScene(scenes.cornell_box(16, 16))
    gen = torch.Generator(device="cuda")
    gen.manual_seed(threads)
    rays = torch.rand((threads, 4099, 8), generator=gen, device="cuda")
    rays[..., 1] *= 2.0
    rays[..., 4:7] -= 0.5
    rays[..., 3], rays[..., 7] = 1e-4, 1000.0
    want = torch.zeros((threads, 4099, 6), dtype=torch.int32, device="cuda")
    got = torch.full_like(want, -1)
    for k in range(threads):
        g.trace(rays[k], want[k])
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(threads)]
    start = threading.Barrier(threads)
    errors = []

    def work(k):
        try:
            torch.cuda.set_device(0)
            start.wait(60)
            for _ in range(8):
                g.trace(rays[k], got[k], stream=streams[k])
        except Exception as e:
            errors.append(e)

    pool = [threading.Thread(target=work, args=(k,)) for k in range(threads)]
    for t in pool:
        t.start()
    for t in pool:
        t.join()
    torch.cuda.synchronize()
    assert not errors
    assert torch.equal(got, want)
