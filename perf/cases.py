"""Performance cases: what a program that uses this framework has it do, each through a public entry point.

listed()             the named cases
draw(rng)            one more case from the ranges that the listed ones stand for
prepare(case, seed)  what the program holds before the call: scene, pipeline, buffers, targets, inputs
run(state)           one pass, and everything it computes
work(case)           bytes and floating-point operations that one pass cannot do without
exact(case, seed)    the pass's results in 64 bits, where they have such a value

The kinds of work:
  render    Pipeline.render: one plain path-traced frame (colour, first-hit normal and albedo)
  trace     GpuScene.trace: ray queries outside a render (picking, probes, visibility)
  restir    a frame of the ReSTIR GI loop: 1-spp render into per-pixel reservoirs, temporal and spatial
            resampling, end-of-frame advance
  resample  the two resampling passes alone, on the reservoirs of a rendered frame
  guided    Pipeline.render with a trained guide network (no online training, which is not repeatable)
  guide     the guide network by itself: evaluation, loss and gradient, Adam steps, evaluation
  batch     Pipeline.batch_render: many small requests as one wavefront

Markov-guided renders are left out: their world grid is updated by racing threads, as in the
reference, so two renders of the same frame differ.
"""
import functools
import math

import numpy as np
import torch

import lambent_b200 as lb
from lambent_b200 import _abi, scenes

QUALITY = {"low": lb.path_tracing.Low, "medium": lb.path_tracing.Medium, "high": lb.path_tracing.High}
# ray segments per sample and floating-point operations per segment (8-wide node tests at 20
# operations a box, triangle tests at 60, shading at 500), as counted on these scenes
SCENES = {"cornell": (3.9, 2000), "textured": (4.0, 2000), "cutout": (4.0, 2500), "occluded": (3.9, 2000),
          "field": (3.5, 5000), "boxes": (4.0, 3500)}


def listed():
    return [
        # the smallest call: an interactive preview of a small scene with the default options' depth
        {"name": "render_preview", "kind": "render", "scene": "cornell", "width": 128, "height": 128, "spp": 1,
         "depth": 5, "quality": "medium"},
        # an ordinary still of a small scene
        {"name": "render_cornell", "kind": "render", "scene": "cornell", "width": 256, "height": 256, "spp": 16,
         "depth": 8, "quality": "medium"},
        # spectral shader, non-uniform textures, alpha-tested geometry, an odd image size
        {"name": "render_cutout_high", "kind": "render", "scene": "cutout", "width": 617, "height": 349, "spp": 4,
         "depth": 8, "quality": "high"},
        # the benchmark's frame: 1.31M triangles in 64 instances, 1080p
        {"name": "render_field_1080p", "kind": "render", "scene": "field", "width": 1920, "height": 1080, "spp": 16,
         "depth": 12, "quality": "medium"},
        # picking and light probes: a thousand rays, latency counts
        {"name": "trace_probes", "kind": "trace", "scene": "field", "rays": 1000, "mode": "closest", "mix": "random"},
        # shadow rays between scattered points of a large scene
        {"name": "trace_shadow", "kind": "trace", "scene": "field", "rays": 300007, "mode": "any", "mix": "random"},
        # a caller's own integrator: camera rays and scattered ones, in large batches
        {"name": "trace_bulk", "kind": "trace", "scene": "field", "rays": 4194304, "mode": "closest", "mix": "camera"},
        # one frame of the ReSTIR GI loop at 1080p
        {"name": "restir_frame_1080p", "kind": "restir", "width": 1920, "height": 1080, "depth": 8, "neighbours": 5,
         "space": 61},
        # the resampling passes with their default options
        {"name": "resample_720p", "kind": "resample", "width": 1280, "height": 720, "neighbours": 8, "space": 61},
        # sampling a trained guide in an indirectly lit room
        {"name": "render_guided", "kind": "guided", "width": 960, "height": 540, "spp": 4, "depth": 8,
         "quality": "medium"},
        # training the guide: the render loop's minibatch, steps per wave and an odd number of queries
        {"name": "guide_training", "kind": "guide", "records": 65536, "batch": 16384, "steps": 32, "queries": 100003},
        # serving thumbnails: 64 requests over four scenes
        {"name": "batch_thumbnails", "kind": "batch", "requests": 64, "width": 128, "height": 128, "spp": 4, "depth": 8},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["render", "render", "render", "trace", "trace", "restir", "resample", "guided", "guide", "batch"])
    quality = rng.choice(["low", "medium", "medium", "high"])
    if kind == "render":
        scene = rng.choice(["cornell", "textured", "cutout", "field"])
        w = _log_int(rng, 64, 1920)
        return {"kind": kind, "scene": scene, "width": w, "height": max(33, w * 9 // 16 + rng.randrange(7)),
                "spp": _log_int(rng, 1, 12), "depth": rng.randint(4, 12 if scene == "field" else 8), "quality": quality}
    if kind == "trace":
        return {"kind": kind, "scene": rng.choice(["field", "field", "cutout"]), "rays": _log_int(rng, 500, 4000000),
                "mode": rng.choice(["closest", "closest", "any"]), "mix": rng.choice(["random", "camera"])}
    if kind in ("restir", "resample"):
        w = _log_int(rng, 320, 1920)
        case = {"kind": kind, "width": w, "height": w * 9 // 16 + rng.randrange(7), "neighbours": rng.randint(3, 10),
                "space": rng.choice([31, 61])}
        return dict(case, depth=rng.randint(5, 8)) if kind == "restir" else case
    if kind == "guided":
        w = _log_int(rng, 160, 1280)
        return {"kind": kind, "width": w, "height": w * 9 // 16 + rng.randrange(7), "spp": rng.randint(1, 4), "depth": 8,
                "quality": quality}
    if kind == "guide":
        return {"kind": kind, "records": _log_int(rng, 4000, 200000), "batch": 128 * _log_int(rng, 16, 256),
                "steps": _log_int(rng, 4, 48), "queries": _log_int(rng, 100, 1000000)}
    w = _log_int(rng, 48, 256)
    return {"kind": kind, "requests": _log_int(rng, 8, 128), "width": w, "height": w + rng.randrange(9),
            "spp": rng.randint(1, 4), "depth": rng.randint(5, 8)}


# ---------------------------------------------------------------- scenes and cameras
@functools.lru_cache(maxsize=None)
def _host_scene(name, variant=0):
    if name == "cornell":
        return scenes.cornell_box()
    if name == "occluded":
        return scenes.occluded_cornell()
    if name == "textured":
        return scenes.textured_cornell()
    if name == "cutout":  # the textured box with holes punched into its textures, alpha tested
        s = scenes.textured_cornell()
        s.blas[0]["flags"] = 0
        rng = np.random.default_rng(3)
        for tex in s.diffuse:
            holes = rng.random(((tex.shape[0] + 7) // 8, (tex.shape[1] + 7) // 8)) < 0.2
            tex[..., 3][np.kron(holes, np.ones((8, 8), bool))[: tex.shape[0], : tex.shape[1]]] = 0
        return s
    if name == "boxes":
        return scenes.box_field((10000, 30000, 90000, 250000)[variant], seed=variant)
    return scenes.icosphere_field()


@functools.lru_cache(maxsize=None)
def _gpu_scene(name, variant=0):
    # a program builds a scene once and renders many frames of it
    return lb.GpuScene(_host_scene(name, variant))


def _camera(name, rng, aspect):
    if name == "field":
        a = rng.uniform(0.0, 2.0 * math.pi)
        return scenes.make_camera((16.0 * math.sin(a), rng.uniform(0.0, 4.0), 16.0 * math.cos(a)), (0.0, 0.0, 0.0), 55.0, aspect)
    return scenes.make_camera((rng.uniform(-0.4, 0.4), rng.uniform(0.8, 1.2), 3.4), (0.0, 1.0, 0.0), 40.0, aspect)


def _targets(w, h):
    return [torch.zeros((h, w, 4), dtype=torch.float32, device="cuda") for _ in range(3)]


def _unit(v):
    return v / v.norm(dim=-1, keepdim=True)


class _Raw:
    """A device buffer of the framework for torch.as_tensor; the tensor keeps this object, and it the owner."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": "<i4", "version": 2}


def _reservoir_views(buffers, which):
    """The lam_reservoir fields as views: floating ones and whole ones apart."""
    ptr, size = buffers.device_buffer(which)
    i = torch.as_tensor(_Raw(buffers, ptr, (size // 64, 16)), device="cuda")
    f = i.view(torch.float32)
    return {"visible_point": f[:, 0:3], "sample_point": f[:, 4:7], "radiance": f[:, 8:11], "roughness_w": f[:, 12:14],
            "weight": f[:, 15], "normal_v": i[:, 3], "normal_s": i[:, 7], "type": i[:, 11], "confidence": i[:, 14]}


# ---------------------------------------------------------------- states
def prepare(case, seed):
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    st = dict(case, frame=int(seed) * 7919 % (1 << 30))
    return {"render": _prepare_render, "trace": _prepare_trace, "restir": _prepare_restir, "resample": _prepare_restir,
            "guided": _prepare_guided, "guide": _prepare_guide, "batch": _prepare_batch}[case["kind"]](st, rng, gen)


def _prepare_render(st, rng, gen):
    host = _host_scene(st["scene"])
    st["gpu"] = _gpu_scene(st["scene"])
    st["camera"] = _camera(st["scene"], rng, st["width"] / st["height"])
    st["pipe"] = lb.RayTracer(QUALITY[st["quality"]]).create_pipeline(*host.layout_counts(), lb.PathTracerOpts(
        samples=st["spp"], restir_temporal=_abi.RESTIR_DISABLED, max_depth=st["depth"]))
    st["buffers"] = lb.DataBuffers(st["width"], st["height"], 1, 0)
    st["images"] = _targets(st["width"], st["height"])
    st["targets"] = lb.targets_from(*st["images"])
    return st


def _prepare_trace(st, rng, gen):
    n = st["rays"]
    st["gpu"] = _gpu_scene(st["scene"])
    r = lambda *s: torch.rand(s, generator=gen, device="cuda")
    span, mid = (12.0, 0.0) if st["scene"] == "field" else (0.95, 1.0)
    origin = (2.0 * r(n, 3) - 1.0) * span
    origin[:, 1] += mid
    if st["mode"] == "any":  # towards another point, as far as it
        target = (2.0 * r(n, 3) - 1.0) * span
        target[:, 1] += mid
        d = target - origin
        far = torch.ones(n, device="cuda")
    else:
        d = _unit(torch.randn((n, 3), generator=gen, device="cuda"))
        far = torch.full((n,), 1000.0, device="cuda")
    if st["mix"] == "camera":  # the first half in image order from one point
        half = n // 2
        side = max(1, math.isqrt(half))
        eye = torch.tensor([0.0, 2.0, 16.0] if st["scene"] == "field" else [0.0, 1.0, 3.4], device="cuda")
        k = torch.arange(half, device="cuda")
        at = torch.stack([(k % side) / side - 0.5, 0.5 - (k // side) / side, torch.full((half,), -0.9, device="cuda")], 1)
        origin[:half] = eye + 0.01 * r(3)
        d[:half] = _unit(at.float())
        far[:half] = 1000.0
    st["ray_tensor"] = torch.cat([origin, torch.full((n, 1), 1e-4, device="cuda"), d, far[:, None]], 1).contiguous()
    st["hits"] = torch.zeros((n, 6), dtype=torch.int32, device="cuda")
    st["hit_floats"] = st["hits"].view(torch.float32)[:, 0:3]
    st["hit_ids"] = st["hits"][:, 3:6]
    st["trace_mode"] = _abi.TRACE_ANY if st["mode"] == "any" else _abi.TRACE_CLOSEST
    return st


def _prepare_restir(st, rng, gen):
    w, h = st["width"], st["height"]
    host = _host_scene("cornell")
    st["gpu"] = _gpu_scene("cornell")
    st["camera"] = _camera("cornell", rng, w / h)
    st["pipe"] = lb.RayTracer(lb.path_tracing.Medium).create_pipeline(*host.layout_counts(), lb.PathTracerOpts(
        samples=1, restir_temporal=_abi.RESTIR_PER_PIXEL, max_depth=st.get("depth", 5)))
    st["buffers"] = lb.DataBuffers(w, h, 1500000, lb.BufferType.all())
    st["images"] = _targets(w, h)
    st["targets"] = lb.targets_from(*st["images"])
    st["advance"] = lb.AdvanceOptions(20)
    if st["kind"] == "restir":
        st["reservoirs"] = _reservoir_views(st["buffers"], lb.DataBuffers.OLD_RESERVOIRS)
        return st
    # reservoirs of two frames: the passes then have a history and a current frame
    for k in range(2):
        st["pipe"].render(st["gpu"], st["buffers"], st["camera"], st["targets"], st["frame"] + k)
        if k == 0:
            st["buffers"].advance_frame(lb.BufferType.all(), st["advance"])
    st["reservoirs"] = _reservoir_views(st["buffers"], lb.DataBuffers.RESERVOIRS)
    return st


def _guide_records(n, gen):
    """Vertices of a room lit through the gap above a plate: positions on its surfaces, directions
    scattered around the light, log-normal weights."""
    r = lambda *s: torch.rand(s, generator=gen, device="cuda")
    g = lambda *s: torch.randn(s, generator=gen, device="cuda")
    pos = torch.stack([2 * r(n) - 1, 2 * r(n), 2 * r(n) - 1], 1)
    axis = torch.randint(0, 5, (n,), generator=gen, device="cuda")
    normals = torch.tensor([[0, 1, 0], [0, -1, 0], [0, 0, 1], [1, 0, 0], [-1, 0, 0]], device="cuda").float()
    normal = normals[axis]
    pos = torch.where(normal != 0, torch.tensor([0.0, 1.0, 0.0], device="cuda") - normal, pos)
    wo = _unit(normal + 0.6 * _unit(g(n, 3)))
    wi = _unit(torch.tensor([0.0, 1.95, 0.0], device="cuda") - pos + 0.3 * g(n, 3))
    return torch.cat([pos, normal, wo, wi, torch.exp(0.5 * g(n, 1))], 1).contiguous()


def _prepare_guided(st, rng, gen):
    w, h = st["width"], st["height"]
    host = _host_scene("occluded")
    st["gpu"] = _gpu_scene("occluded")
    st["camera"] = _camera("occluded", rng, w / h)
    st["pipe"] = lb.RayTracer(QUALITY[st["quality"]]).create_pipeline(*host.layout_counts(), lb.PathTracerOpts(
        samples=st["spp"], restir_temporal=_abi.RESTIR_DISABLED, max_depth=st["depth"], guide_mode=lb.GuideMode.LEARNED))
    st["guide"] = lb.Guide(lb.GuideOptions(train_spp=0, record_capacity=0, seed=1 + st["frame"] % 1000))
    st["guide"].train(_guide_records(65536, gen), 48, st["gpu"].bounds())
    st["pipe"].set_guide(st["guide"])
    st["buffers"] = lb.DataBuffers(w, h, 1, 0)
    st["images"] = _targets(w, h)
    st["targets"] = lb.targets_from(*st["images"])
    return st


ROOM = [-1.0, 0.0, -1.0, 1.0, 2.0, 1.0]


def _guide_params(gen):
    """Weights as a trained network has them, representable in BF16, the type the network computes in."""
    p = torch.randn((4, 64, 64), generator=gen, device="cuda") * 0.17
    p[:3, 63] = 0.0
    p[3, 40:] = 0.0
    return p.bfloat16().float()


def _prepare_guide(st, rng, gen):
    n = st["records"]
    st["guide"] = lb.Guide(lb.GuideOptions(batch=st["batch"], record_capacity=0, seed=1 + st["frame"] % 1000))
    st["params"] = _guide_params(gen)
    st["guide"].set_params(st["params"].reshape(-1).tolist())
    st["record_tensor"] = _guide_records(n, gen)
    st["query_tensor"] = _guide_records(st["queries"], gen)[:, :9].contiguous()
    st["before"] = torch.zeros((st["queries"], 40), dtype=torch.float32, device="cuda")
    st["after"] = torch.zeros_like(st["before"])
    st["grad"] = torch.zeros(16384, dtype=torch.float32, device="cuda")
    st["loss"] = torch.zeros(1, dtype=torch.float32, device="cuda")
    return st


def _prepare_batch(st, rng, gen):
    w, h = st["width"], st["height"]
    hosts = [_host_scene("boxes", v) for v in range(4)]
    counts = [max(c) for c in zip(*(s.layout_counts() for s in hosts))]
    st["pipe"] = lb.RayTracer(lb.path_tracing.Medium).create_pipeline(*counts, lb.PathTracerOpts(
        restir_temporal=_abi.RESTIR_DISABLED, max_depth=st["depth"]))
    st["image"] = torch.zeros((st["requests"], h, w, 4), dtype=torch.float32, device="cuda")
    st["list"] = [(_gpu_scene("boxes", k % 4), _camera("boxes", rng, w / h), lb.targets_from(st["image"][k]),
                   1 + (st["spp"] + k) % st["spp"] if st["spp"] > 1 else 1, st["frame"] + k) for k in range(st["requests"])]
    return st


# ---------------------------------------------------------------- passes
def run(st):
    kind = st["kind"]
    if kind in ("render", "guided"):
        st["pipe"].render(st["gpu"], st["buffers"], st["camera"], st["targets"], st["frame"])
        return st["images"]
    if kind == "trace":
        st["gpu"].trace(st["ray_tensor"], st["hits"], st["trace_mode"])
        return {"tuv": st["hit_floats"], "ids": st["hit_ids"]}
    if kind in ("restir", "resample"):
        b, k = st["buffers"], st["frame"]
        st["frame"] = k + 1
        if kind == "restir":
            st["pipe"].render(st["gpu"], b, st["camera"], st["targets"], k)
        b.temporal_resampling(k)
        b.spatial_resampling(st["targets"], st["neighbours"], st["space"], k)
        if kind == "restir":
            b.advance_frame(lb.BufferType.all(), st["advance"])
        return {"images": st["images"], "reservoirs": st["reservoirs"]}
    if kind == "guide":
        g = st["guide"]
        g.eval(st["query_tensor"], ROOM, st["before"])
        g.loss_grad(st["record_tensor"], ROOM, st["grad"], st["loss"])
        g.train(st["record_tensor"], st["steps"], ROOM)
        g.eval(st["query_tensor"], ROOM, st["after"])
        return {"before": st["before"], "grad": st["grad"], "loss": st["loss"], "after": st["after"]}
    st["pipe"].batch_render(st["list"])
    return st["image"]


# ---------------------------------------------------------------- what a pass cannot do without
def work(case):
    kind = case["kind"]
    if kind == "trace":
        return {"bytes": 56.0 * case["rays"], "flops": float(SCENES[case["scene"]][1] * case["rays"])}
    if kind == "guide":
        layers = 2.0 * 4 * 64 * 64
        return {"bytes": 392.0 * case["queries"] + 52.0 * case["records"] + 131072.0 * case["steps"],
                "flops": layers * (2 * case["queries"] + 3 * case["records"] + 3 * case["batch"] * case["steps"])}
    pixels = case["width"] * case["height"] * case.get("requests", 1)
    passes = 320.0 + 64.0 * case.get("neighbours", 0)  # reservoirs in and out, neighbours, surface record, image
    if kind == "resample":
        return {"bytes": passes * pixels, "flops": 1000.0 * pixels}
    segments, flops = SCENES[{"restir": "cornell", "guided": "occluded", "batch": "boxes"}.get(kind) or case["scene"]]
    rays = pixels * case.get("spp", 1) * min(segments, case["depth"])
    out = {"bytes": 48.0 * pixels, "flops": flops * rays}
    if kind == "batch":
        out = {"bytes": 16.0 * pixels, "flops": flops * rays * (case["spp"] + 1) / (2.0 * case["spp"])}
    elif kind == "restir":
        out["bytes"] += (passes + 320.0) * pixels + 168.0 * 1500000
    elif kind == "guided":
        out["flops"] += 0.5 * rays * 2.0 * 4 * 64 * 64
    return out


# ---------------------------------------------------------------- results in 64 bits
def exact(case, seed):
    if case["kind"] == "trace" and case["mode"] == "closest" and case["rays"] <= 4096 and case["scene"] == "field":
        return {"tuv": _exact_hits(prepare(case, seed)), "ids": None}
    if case["kind"] == "guide":
        return _exact_guide(prepare(case, seed))
    return None  # a path's decisions hang on the last bits of 32-bit arithmetic


def _exact_hits(st):
    """Closest hits by testing every triangle of every instance whose bounding sphere a ray meets."""
    host = _host_scene(st["scene"])
    rays = st["ray_tensor"].double()
    o, d, tmin, tmax = rays[:, 0:3], rays[:, 4:7], rays[:, 3], rays[:, 7]
    best = torch.zeros((o.shape[0], 3), dtype=torch.float64, device="cuda")
    far = tmax.clone()
    for inst in host.instances:
        blas = host.blas[inst["blas"]]
        m = torch.tensor(np.asarray(inst["transform"], np.float64).reshape(3, 4), device="cuda")
        inv = torch.linalg.inv(m[:, :3])
        v = torch.tensor(blas["vertices"][:, :3], device="cuda").double()[torch.tensor(blas["indices"].astype(np.int64), device="cuda")].reshape(-1, 3, 3)
        oo, od = (o - m[:, 3]) @ inv.T, d @ inv.T
        near = torch.linalg.cross(oo, od).norm(dim=1) <= v.norm(dim=2).max() * od.norm(dim=1) * (1.0 + 1e-9)
        pick = near.nonzero()[:, 0]
        e1, e2 = v[:, 1] - v[:, 0], v[:, 2] - v[:, 0]
        for part in pick.split(256):
            a, b = oo[part][:, None], od[part][:, None]
            p = torch.linalg.cross(b.expand(-1, e2.shape[0], -1), e2[None].expand(len(part), -1, -1))
            det = (p * e1).sum(-1)
            s = a - v[None, :, 0]
            q = torch.linalg.cross(s, e1[None].expand_as(s))
            u, w, t = (s * p).sum(-1) / det, (b * q).sum(-1) / det, (e2 * q).sum(-1) / det
            ok = (u >= 0) & (w >= 0) & (u + w <= 1) & (t > tmin[part, None]) & (t < far[part, None])
            t, k = torch.where(ok, t, math.inf).min(dim=1)
            hit = t < far[part]
            row = torch.arange(len(part), device="cuda")
            got = torch.stack([t, u[row, k], w[row, k]], 1)
            best[part] = torch.where(hit[:, None], got, best[part])
            far[part] = torch.where(hit, t, far[part])
    return best


def _exact_guide(st):
    """Head outputs, loss and gradient of the network at the weights it starts from."""
    box = torch.tensor(ROOM, dtype=torch.float64, device="cuda")

    def features(q):
        q = q.double()
        u = ((q[:, 0:3] - box[:3]) / (box[3:] - box[:3])).clamp(0.0, 1.0)
        f = [torch.stack([torch.sin(2.0 ** k * math.pi * u), torch.cos(2.0 ** k * math.pi * u)], 2).flatten(1) for k in range(5)]
        d = q[:, 3:9]
        f += [d, torch.stack([g(k * math.pi * d) for k in (1, 2) for g in (torch.sin, torch.cos)], 2).flatten(1)]
        return torch.cat(f + [torch.zeros_like(d[:, :3]), torch.ones_like(d[:, :1])], 1)

    def heads(w, x):
        for layer in range(3):
            x = torch.relu(x @ w[layer].T)
            x = torch.cat([x[:, :63], torch.ones_like(x[:, :1])], 1)
        return (x @ w[3].T)[:, :40]

    w = st["params"].double().requires_grad_(True)
    rec = st["record_tensor"].double()
    raw = heads(w, features(rec[:, :9]))
    kappa = raw[:, 8:16].clamp(-3.0, 6.0).exp()
    mean = torch.nn.functional.normalize(torch.stack([raw[:, 16:24], raw[:, 24:32], raw[:, 32:40]], 2), dim=2)
    log_q = torch.logsumexp(torch.log_softmax(raw[:, 0:8], 1) + torch.log(kappa) - math.log(2.0 * math.pi)
                            - torch.log1p(-torch.exp(-2.0 * kappa)) + kappa * ((mean * rec[:, None, 9:12]).sum(2) - 1.0), 1)
    loss = -(rec[:, 12] * log_q).mean()
    grad = torch.autograd.grad(loss, w)[0]
    grad[:3, 63] = 0.0
    grad[3, 40:] = 0.0
    with torch.no_grad():
        before = heads(w, features(st["query_tensor"]))
    return {"before": before, "grad": grad.reshape(-1), "loss": loss.detach().reshape(1), "after": None}
