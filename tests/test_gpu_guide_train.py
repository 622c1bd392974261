"""Runs of Adam steps in one launch: the result does not depend on how the steps are split over calls
and launches (at most 64 steps each), on one tile or several per CTA, or on being replayed from a
CUDA graph.  Evaluation: a query's outputs do not depend on the queries beside it, nor on the output's
alignment."""
import pytest

import lambent_b200 as lb

pytestmark = pytest.mark.gpu

BOX = [-1.0, 0.0, -1.0, 1.0, 2.0, 1.0]


def records(n, seed):
    import torch
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    r = torch.randn((n, 13), generator=gen, device="cuda")
    r[:, 3:6], r[:, 6:9], r[:, 9:12] = (v / v.norm(dim=1, keepdim=True) for v in (r[:, 3:6], r[:, 6:9], r[:, 9:12]))
    r[:, 12] = r[:, 12].abs()
    return r.contiguous()


@pytest.mark.parametrize("batch,n,split", [(128, 1, [1, 2]), (128 * 148, 5000, [3, 4]), (128 * 149, 5000, [5]),
                                           (128 * 300, 70000, [1, 1, 1]), (1024, 777, [64, 1, 70])])
def test_steps_split_over_calls(cuda, batch, n, split):
    import torch
    rec = records(n, batch)
    got = []
    for parts in ([1] * sum(split), split):
        g = lb.Guide(lb.GuideOptions(batch=batch, record_capacity=0, seed=3))
        for k in parts:
            g.train(rec, k, BOX)
        torch.cuda.synchronize()
        assert g.progress() == (sum(split), 0)
        got.append(torch.tensor(g.params()))
    assert torch.isfinite(got[0]).all()
    assert torch.equal(got[0], got[1])


def test_training_in_a_graph(cuda):
    import torch
    rec = records(4096, 1)
    g = lb.Guide(lb.GuideOptions(batch=2048, record_capacity=0, seed=3))
    start = g.params()
    g.train(rec, 5, BOX)
    want = torch.tensor(g.params())
    g.set_params(start)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        g.train(rec, 5, BOX)
    assert torch.equal(torch.tensor(g.params()), torch.tensor(start))  # captured, not run
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(torch.tensor(g.params()), want)


@pytest.mark.parametrize("n", [1, 127, 128, 129, 255, 256, 257, 511, 513, 1025, 200003])
def test_eval_edges(cuda, n):
    import torch
    g = lb.Guide(lb.GuideOptions(record_capacity=0, seed=n))
    q = records(n, n)[:, :9].contiguous()
    whole = torch.full((n, 40), -7.0, device="cuda")
    g.eval(q, BOX, whole)
    store = torch.full((n * 40 + 3,), -7.0, device="cuda")
    for offset in (1, 2):  # rows of the output 4 and 8 bytes off 16-byte alignment
        odd = store[offset:offset + n * 40].view(n, 40)
        g.eval(q, BOX, odd)
        assert torch.equal(odd, whole)
    for k in {0, n // 2, max(0, n - 1)}:
        one = torch.empty((1, 40), device="cuda")
        g.eval(q[k:k + 1].contiguous(), BOX, one)
        assert torch.equal(one[0], whole[k])
    assert g.progress() == (0, 0)
