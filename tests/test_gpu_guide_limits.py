"""Training whose waits give up: a step is taken by all thread blocks or by none, whichever wait it was
and wherever the others were."""
import numpy as np
import pytest

import lambent_b200 as lb
from lambent_b200 import _abi

pytestmark = pytest.mark.gpu

BOX = [-1.0, 0.0, -1.0, 1.0, 2.0, 1.0]


def records(n):
    import torch
    gen = torch.Generator(device="cuda")
    gen.manual_seed(n)
    r = torch.randn((n, 13), generator=gen, device="cuda")
    r[:, 3:6], r[:, 6:9], r[:, 9:12] = (v / v.norm(dim=1, keepdim=True) for v in (r[:, 3:6], r[:, 6:9], r[:, 9:12]))
    r[:, 12] = r[:, 12].abs()
    return r.contiguous()


@pytest.mark.parametrize("batch", [128, 128 * 148, 128 * 300])
def test_training_that_gives_up_takes_no_step(cuda, batch):
    """With momentum from earlier steps, a step on zero gradients would move the parameters."""
    import torch
    rec = records(5000)
    g = lb.Guide(lb.GuideOptions(batch=batch, record_capacity=0, seed=3))
    g.train(rec, 3, BOX)
    before = np.array(g.params())
    assert g.progress() == (3, 0)
    g.set_wait_limit(0)
    g.train(rec, 70, BOX)  # two launches
    torch.cuda.synchronize()
    with pytest.raises(lb.LambentError) as e:
        g.progress()
    assert e.value.code == _abi.ERR_DEVICE_TIMEOUT
    g.progress()  # reported once
    np.testing.assert_array_equal(np.array(g.params()), before)
    g.set_wait_limit(1 << 20)
    fresh = lb.Guide(lb.GuideOptions(batch=batch, record_capacity=0, seed=3))
    for x in (g, fresh):
        x.set_params(list(before))
        x.train(rec, 5, BOX)
    torch.cuda.synchronize()
    np.testing.assert_array_equal(np.array(g.params()), np.array(fresh.params()))
    assert g.progress() == fresh.progress() == (5, 0)


def test_parameters_are_always_those_of_whole_steps(cuda):
    """Limits at which some waits give up and others do not."""
    import torch
    rec = records(5000)
    opts = lb.GuideOptions(batch=128 * 148, record_capacity=0, seed=3)
    whole = [np.array(lb.Guide(opts).params())]
    for steps in range(1, 7):
        g = lb.Guide(opts)
        g.train(rec, steps, BOX)
        whole.append(np.array(g.params()))
        assert g.progress() == (steps, 0)
    gave_up = 0
    for limit in [1, 2, 3, 5, 8, 13, 21, 34, 55, 144, 1000] * 4:
        g = lb.Guide(opts)
        g.set_wait_limit(limit)
        g.train(rec, 6, BOX)
        torch.cuda.synchronize()
        p = np.array(g.params())
        taken = [k for k in range(7) if np.array_equal(p, whole[k])]
        assert taken, limit
        try:
            g.progress()
            assert taken == [6]
        except lb.LambentError as e:
            assert e.code == _abi.ERR_DEVICE_TIMEOUT
            gave_up += 1
    assert gave_up


def test_launch_count_of_a_training_render(cuda):
    """A launch takes at most 64 Adam steps; kernel_launches counts each."""
    import torch
    from lambent_b200 import scenes
    s = scenes.cornell_box(64, 64)
    g = lb.GpuScene(s)
    count = {}
    for steps in (0, 1, 64, 65, 200):
        guide = lb.Guide(lb.GuideOptions(steps_per_wave=steps, batch=128, record_capacity=4096, train_spp=2))
        pipe = lb.RayTracer(lb.path_tracing.Medium).create_pipeline(*s.layout_counts(), lb.PathTracerOpts(
            samples=2, restir_temporal=_abi.RESTIR_DISABLED, max_depth=3, guide_mode=_abi.GUIDE_LEARNED))
        pipe.set_guide(guide)
        col = torch.zeros((64, 64, 4), device="cuda")
        pipe.render(g, lb.DataBuffers(64, 64, 1, 0), s.camera, lb.targets_from(col), 0)
        torch.cuda.synchronize()
        assert guide.progress()[0] == steps
        count[steps] = pipe.stats().kernel_launches
    assert [count[k] - count[0] for k in (1, 64, 65, 200)] == [1, 1, 2, 4]


@pytest.mark.parametrize("batch", [128 * 100, 128 * 148])
def test_guides_trained_in_two_streams(cuda, batch):
    """Each launch fills most of the device with blocks that wait for one another: two at a time run, one
    after the other or side by side, and neither waits for blocks that cannot start."""
    import torch
    rec = records(5000)
    opts = lb.GuideOptions(batch=batch, record_capacity=0, seed=3)
    want = lb.Guide(opts)
    for _ in range(8):
        want.train(rec, 8, BOX)
    torch.cuda.synchronize()
    guides, streams = [lb.Guide(opts) for _ in range(2)], [torch.cuda.Stream() for _ in range(2)]
    for g in guides:
        g.set_wait_limit(1 << 16)  # a second or two, should they hold each other up
    for _ in range(8):
        for g, st in zip(guides, streams):
            g.train(rec, 8, BOX, stream=st)
    torch.cuda.synchronize()
    for g in guides:
        assert g.progress() == (64, 0)
        np.testing.assert_array_equal(np.array(g.params()), np.array(want.params()))
