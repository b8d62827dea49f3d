"""The measured workloads: closest-hit batches, renders with each estimator, batched renders, the
denoiser, the radiance cache's inference and training, and .hdr output, each through the public
entry points of pico_gb300.

A case is a dict of plain values; `kind` selects the entry point.  One context serves the process,
as in a program that renders: the scene, rays, queries and buffers of a case belong to its state.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

import pico_gb300
from pico_gb300 import scenes

PIXELS_1080P = 1920 * 1080
_context = None


def _ctx():
    global _context
    if _context is None:
        _context = pico_gb300.Context(0)
    return _context


def listed():
    return [
        # a picking or probe query of an interactive program: a few rays, where the call itself counts
        dict(name="trace_1k", kind="trace", n=1000, instances=64, level=2, host=False),
        # a mid-sized batch handed over as a numpy array, ragged, copies included
        dict(name="trace_host_300k", kind="trace", n=300007, instances=4096, level=4, host=True),
        # the traversal benchmark: half coherent primary rays, half cosine bounces, 21M instanced triangles
        dict(name="trace_16m", kind="trace", n=1 << 24, instances=4096, level=4, host=False),
        # the small full render that the CPU reference runs too: host buffers in and out, denoised, tone mapped
        dict(name="render_cornell_256", kind="render", scene="cornell", instances=8, width=256, height=256, spp=16,
             depth=5, estimator=0, denoise=True, tonemap=True, host=True),
        # the headline render on device buffers
        dict(name="render_field_1080p", kind="render", scene="field", instances=4096, width=1920, height=1080, spp=64,
             depth=8, estimator=0, denoise=True, tonemap=False, host=False),
        # the physical estimator on a sky-and-sun scene with mirrors, an odd image size, host buffers
        dict(name="render_physical_853x479", kind="render", scene="glossy", instances=200, width=853, height=479,
             spp=16, depth=8, estimator=1, denoise=False, tonemap=False, host=True),
        # the radiance cache, trained while it renders: the passes of a preview frame
        dict(name="render_cache_540p", kind="cache", instances=1024, width=960, height=540, spp=4, depth=8,
             log2_table=19),
        # renders of uneven size, scene, samples and depth in one graph launch
        dict(name="render_batch_6", kind="batch", renders=6, mix=5, scale=1.0),
        # the denoiser on a full frame's G-buffer in device memory
        dict(name="denoise_1080p", kind="denoise", width=1920, height=1080, sky=0),
        # one frame's cache queries: second path vertices in pixel order
        dict(name="infer_1m", kind="infer", n=1000003, log2_table=19),
        # one optimiser step on the default batch and table, gradients fetched
        dict(name="train_64k", kind="train", n=65536, log2_table=19),
        # writing a full frame: RGBE and run-length coding of a host image
        dict(name="hdr_1080p", kind="hdr", width=1920, height=1080),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["trace", "trace", "render", "render", "cache", "batch", "denoise", "infer", "train", "hdr"])
    if kind == "trace":
        host = rng.random() < 0.4
        return dict(kind=kind, n=_log_int(rng, 500, 2e6 if host else 1.6e7), instances=_log_int(rng, 64, 4096),
                    level=rng.choice([2, 3, 4]), host=host)
    if kind == "render":
        w = _log_int(rng, 64, 1600)
        h = min(1080, max(48, int(w * rng.uniform(0.5, 1.0))))
        spp = max(1, min(64, _log_int(rng, 4, 64), PIXELS_1080P * 16 // (w * h)))
        scene = rng.choice(["cornell", "field", "glossy"])
        inst = {"cornell": 8, "field": _log_int(rng, 64, 4096), "glossy": _log_int(rng, 20, 200)}[scene]
        return dict(kind=kind, scene=scene, instances=inst, width=w, height=h, spp=spp, depth=rng.randint(3, 8),
                    estimator=rng.choice([0, 1]), denoise=rng.random() < 0.5, tonemap=rng.random() < 0.3,
                    host=rng.random() < 0.5)
    if kind == "cache":
        return dict(kind=kind, instances=_log_int(rng, 64, 1024), width=_log_int(rng, 200, 960),
                    height=_log_int(rng, 120, 540), spp=rng.randint(1, 4), depth=rng.randint(4, 8),
                    log2_table=rng.randint(14, 19))
    if kind == "batch":
        return dict(kind=kind, renders=rng.randint(2, 6), mix=rng.randint(6, 1000), scale=rng.uniform(0.3, 0.9))
    if kind == "denoise":
        return dict(kind=kind, width=_log_int(rng, 65, 1920), height=_log_int(rng, 40, 1080), sky=rng.randint(0, 1))
    if kind == "infer":
        return dict(kind=kind, n=_log_int(rng, 1000, 1e6), log2_table=rng.randint(14, 19))
    if kind == "train":
        return dict(kind=kind, n=_log_int(rng, 2000, 65536), log2_table=rng.randint(14, 19))
    return dict(kind="hdr", width=_log_int(rng, 65, 1920), height=_log_int(rng, 40, 1080))


# ------------------------------------------------------------------------------- inputs
def _generator(seed):
    return torch.Generator("cuda").manual_seed(int(seed) * 7919 + 13)


def _uniform(g, lo, hi, *shape):
    return torch.rand(*shape, generator=g, device="cuda") * (hi - lo) + lo


def _unit(v):
    return v / v.norm(dim=-1, keepdim=True)


def _cosine(g, n):
    """Cosine-distributed directions about the unit normals n."""
    u = torch.rand(len(n), 2, generator=g, device="cuda")
    r, phi = u[:, 0].sqrt(), 2.0 * math.pi * u[:, 1]
    flip = n[:, 2:3].abs() < 0.9
    helper = torch.where(flip, n.new_tensor([[0.0, 0.0, 1.0]]), n.new_tensor([[1.0, 0.0, 0.0]]))
    t = _unit(torch.linalg.cross(n, helper))
    b = torch.linalg.cross(n, t)
    z = (1.0 - u[:, 0]).clamp_min(1e-6).sqrt()
    return _unit((r * phi.cos())[:, None] * t + (r * phi.sin())[:, None] * b + z[:, None] * n)


def _rays(scene, n, seed):
    """Half a centred band of a square pinhole's jittered pixels, half cosine rays off random surface points."""
    g = _generator(seed)
    rays = torch.zeros(n, 8, device="cuda")
    half = n // 2
    side = max(2, int(math.ceil(math.sqrt(2.0 * max(half, 1)))))
    first = (side - max(1, half // side)) // 2 * side
    for a in range(0, half, 1 << 22):
        k = torch.arange(a, min(half, a + (1 << 22)), device="cuda")
        p = k + first
        xi = torch.rand(len(k), 2, generator=g, device="cuda") * 0.5
        dx = ((p % side) + xi[:, 0]) / side - 0.5
        dy = ((p // side) + xi[:, 1]) / side - 0.5
        rays[a:a + len(k), :3] = rays.new_tensor([0.0, 0.0, -130.0])
        rays[a:a + len(k), 4:7] = _unit(torch.stack([-dx, dy, torch.ones_like(dx)], 1))
    m = torch.from_numpy(np.stack([np.asarray(i.transform).reshape(4, 4).T for i in scene.instances])).cuda()
    mesh = scene.meshes[0]
    pos, nrm = torch.from_numpy(mesh.positions).cuda(), torch.from_numpy(mesh.normals).cuda()
    idx = torch.from_numpy(mesh.indices.astype(np.int64)).cuda()
    for a in range(half, n, 1 << 22):
        c = min(n - a, 1 << 22)
        inst = torch.randint(len(m), (c,), generator=g, device="cuda")
        tri = idx[torch.randint(len(idx), (c,), generator=g, device="cuda")]
        u = torch.rand(c, 2, generator=g, device="cuda")
        su = u[:, 0].sqrt()
        w = torch.stack([1.0 - su, u[:, 1] * su, su - u[:, 1] * su], 1)[:, :, None]
        o, q = (w * pos[tri]).sum(1), (w * nrm[tri]).sum(1)
        o = (m[inst, :3, :3] @ o[:, :, None])[:, :, 0] + m[inst, :3, 3]
        q = _unit((m[inst, :3, :3] @ q[:, :, None])[:, :, 0])
        rays[a:a + c, :3] = o + 0.01 * q
        rays[a:a + c, 4:7] = _cosine(g, q)
    rays[:, 3] = 1.0
    rays[:, 7] = 10000.0
    return rays


def _balls(g, k=40):
    """A still life of k balls on a floor for the screen-space inputs: centres, radii, albedos."""
    r = _uniform(g, 0.15, 0.8, k)
    c = torch.stack([_uniform(g, -5.0, 5.0, k), r - 2.0 + _uniform(g, 0.0, 3.0, k) * (r < 0.4), _uniform(g, 4.0, 12.0, k)], 1)
    return c, r, _uniform(g, 0.1, 0.9, k, 3)


def _cast(balls, o, d):
    """Nearest ball or the floor y = -2 (out to 30) along rays: distance (inf: nothing), normal, albedo."""
    c, r, alb = balls
    t = torch.full_like(o[:, 0], math.inf)
    nrm, out = -d.clone(), torch.zeros_like(o)
    tf = (-2.0 - o[:, 1]) / d[:, 1]
    p = o + tf[:, None] * d
    ok = (tf > 1e-3) & (p.abs().amax(1) < 30.0)
    t = torch.where(ok, tf, t)
    nrm[ok] = nrm.new_tensor([0.0, 1.0, 0.0])
    out[ok] = 0.5
    for k in range(len(r)):
        m = o - c[k]
        b, q = (m * d).sum(1), (m * m).sum(1) - r[k] * r[k]
        disc = b * b - q
        tk = -b - disc.clamp_min(0.0).sqrt()
        ok = (disc > 0.0) & (tk > 1e-3) & (tk < t)
        t = torch.where(ok, tk, t)
        nrm = torch.where(ok[:, None], (m + tk[:, None] * d) / r[k], nrm)
        out = torch.where(ok[:, None], alb[k], out)
    return t, nrm, out


def _screen(balls, w, h):
    i = torch.arange(w * h, device="cuda")
    x, y = ((i % w) + 0.5) / w - 0.5, 0.5 - ((i // w) + 0.5) / h
    d = _unit(torch.stack([x * (w / h), y, torch.ones_like(x)], 1))
    t, n, alb = _cast(balls, torch.zeros_like(d), d)
    return d, t, n, alb


def _frame(case, seed):
    """A noisy frame and its G-buffer (colour, normals, positions, albedo), (H, W, 3) each."""
    g = _generator(seed)
    w, h = case["width"], case["height"]
    d, t, n, alb = _screen(_balls(g), w, h)
    hit = torch.isfinite(t)[:, None]
    sky = d.new_tensor([0.10, 0.15, 0.25]) * case.get("sky", 1)
    alb = torch.where(hit, alb, sky)
    pos = torch.where(hit, d * t[:, None].nan_to_num(posinf=0.0), d * 10000.0)
    light = _unit(d.new_tensor([0.4, 0.8, -0.4]))
    shade = (n @ light).clamp_min(0.0)[:, None] * 2.0 + 0.1
    noise = torch.rand(w * h, 3, generator=g, device="cuda").clamp_min(1e-6).log().neg()
    pix = torch.where(hit, alb * shade * noise, sky)
    lamp = (torch.rand(w * h, 1, generator=g, device="cuda") < 1e-4) & hit
    pix = torch.where(lamp, pix + 20.0, pix)
    return [v.reshape(h, w, 3).contiguous() for v in (pix, n, pos, alb)]


def _queries(n, seed):
    """Second path vertices in pixel order, as (n, 16) query records, and radiance targets (n, 4)."""
    g = _generator(seed)
    balls = _balls(g)
    w = max(8, int(math.sqrt(2.0 * n)))
    d, t, nrm, _ = _screen(balls, w, max(8, 3 * n // w))
    keep = torch.isfinite(t)
    d, t, nrm = d[keep], t[keep], nrm[keep]
    o = d * t[:, None] + 0.01 * nrm
    b = _cosine(g, nrm)
    t2, n2, a2 = _cast(balls, o, b)
    keep = torch.isfinite(t2)
    p, v, n2, a2 = (o + t2[:, None] * b)[keep], -b[keep], n2[keep], a2[keep]
    k = torch.arange(n, device="cuda") % len(p)
    q = torch.zeros(n, 16, device="cuda")
    q[:, 0:3], q[:, 3:6], q[:, 6:9], q[:, 10:13] = p[k], v[k], n2[k], a2[k]
    q[:, 9] = _uniform(g, 0.05, 1.0, n)
    target = torch.zeros(n, 4, device="cuda")
    target[:, :3] = a2[k] * torch.rand(n, 3, generator=g, device="cuda").clamp_min(1e-6).log().neg()
    return q, target


BOUNDS = ((-30.0, -2.1, -30.0), (30.0, 4.0, 30.0))


def _network(case, seed):
    """Network (6, 64, 64) and grid (16, T, 2) of a cache that has learnt something."""
    g = _generator(seed + 1)
    mlp = torch.zeros(6, 64, 64, device="cuda")
    for l in range(6):
        rows = 64 if l < 5 else 3
        a = math.sqrt(6.0 / (64 + rows))
        mlp[l, :rows] = _uniform(g, -a, a, rows, 64)
    return mlp, _uniform(g, -0.5, 0.5, 16, 1 << case["log2_table"], 2)


def _scene(case, seed):
    if case["scene"] == "cornell":
        return scenes.cornell_box(), scenes.cornell_camera(case["width"], case["height"])
    if case["scene"] == "glossy":
        return (scenes.glossy_field(n_instances=case["instances"], seed=seed % 100000 + 1),
                scenes.glossy_field_camera(case["width"], case["height"]))
    return (scenes.lit_field(n_instances=case["instances"], seed=seed % 100000 + 1),
            scenes.lit_field_camera(case["width"], case["height"]))


def _batch(case):
    """(width, height, spp, depth, instances) of a batch's renders."""
    rng = np.random.default_rng(case["mix"])
    out = []
    for _ in range(case["renders"]):
        w, h = scenes.BATCH_RESOLUTIONS[rng.integers(len(scenes.BATCH_RESOLUTIONS))]
        out.append((max(8, int(w * case["scale"])), max(8, int(h * case["scale"])),
                    int(scenes.BATCH_SPP[rng.integers(2)]), int(rng.integers(4, 9)),
                    int(round(math.exp(rng.uniform(math.log(64), math.log(1024)))))))
    return out


# ------------------------------------------------------------------------------- states
def prepare(case, seed):
    ctx, kind = _ctx(), case["kind"]
    s = dict(case=case, seed=int(seed), ctx=ctx)
    if kind == "trace":
        scene = scenes.instance_field(n_instances=case["instances"], level=case["level"], seed=seed % 100000 + 1)
        rays = _rays(scene, case["n"], seed)
        s["gs"] = ctx.upload(scene)
        if case["host"]:
            s["rays"] = rays.cpu().numpy()
        else:
            s["rays"] = rays
            s["hits"] = torch.empty(case["n"], 5, dtype=torch.int32, device="cuda")
    elif kind == "render":
        scene, s["camera"] = _scene(case, seed)
        s["gs"] = ctx.upload(scene)
    elif kind == "cache":
        scene, s["camera"] = _scene(dict(case, scene="field"), seed)
        s["gs"] = ctx.upload(scene)
        s["cache"] = pico_gb300.RadianceCache(ctx, log2_table_size=case["log2_table"], seed=seed + 1)
    elif kind == "batch":
        s["gs"] = [ctx.upload(scenes.lit_field(n_instances=b[4], level=3, seed=seed % 100000 + k))
                   for k, b in enumerate(_batch(case))]
    elif kind == "denoise":
        s["inputs"] = _frame(case, seed)
        s["out"] = torch.empty_like(s["inputs"][0])
    elif kind in ("infer", "train"):
        s["queries"], s["targets"] = _queries(case["n"], seed)
        cache = pico_gb300.RadianceCache(ctx, log2_table_size=case["log2_table"], aabb_min=BOUNDS[0],
                                         aabb_max=BOUNDS[1])
        mlp, grid = _network(case, seed)
        cache.set_params(mlp.cpu().numpy(), grid.cpu().numpy())
        s["cache"] = cache
        if kind == "infer":
            s["rgb"] = torch.empty(case["n"], 3, device="cuda")
        else:
            s["grads"] = [torch.empty(6, 64, 64).pin_memory(), torch.empty(16, 1 << case["log2_table"], 2).pin_memory()]
    else:
        s["image"] = _frame(case, seed)[0].cpu().numpy()
        s["file"] = np.zeros(ctx.lib.pico_gpu_hdr_bound(case["width"], case["height"]), np.uint8)
        s["length"] = ctypes.c_size_t(0)
    return s


def run(s):
    case, ctx, kind = s["case"], s["ctx"], s["case"]["kind"]
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "trace":
        if case["host"]:
            h = s["gs"].trace_closest(s["rays"])
            return [h[k] for k in ("inst", "prim", "t", "u", "v")]
        hits = s["hits"]
        s["gs"].trace_closest_device(s["rays"].data_ptr(), case["n"], hits.data_ptr(), stream)
        return [hits[:, 0], hits[:, 1]] + [hits[:, k].view(torch.float32) for k in (2, 3, 4)]
    if kind == "render":
        w, h = case["width"], case["height"]
        opts = dict(seed=s["seed"] + 1, denoise=case["denoise"], tonemap=case["tonemap"], estimator=case["estimator"])
        if case["host"]:
            return list(s["gs"].render(s["camera"], case["depth"], case["spp"], **opts))
        pix, var = torch.zeros(h, w, 3, device="cuda"), torch.zeros(h, w, 3, device="cuda")
        count = torch.zeros(h, w, dtype=torch.int32, device="cuda")
        s["gs"].render_device(s["camera"], case["depth"], case["spp"], pix.data_ptr(), count.data_ptr(),
                              var.data_ptr(), stream, **opts)
        return [pix, count, var]
    if kind == "cache":
        s["cache"].attach()
        return list(s["gs"].render(s["camera"], case["depth"], case["spp"], seed=s["seed"] + 1,
                                   estimator=pico_gb300.ESTIMATOR_RADIANCE_CACHE))
    if kind == "batch":
        items = []
        for k, (gs, (w, h, spp, depth, _)) in enumerate(zip(s["gs"], _batch(case))):
            items.append({"gpu_scene": gs, "camera": scenes.lit_field_camera(w, h), "max_samples": spp,
                          "max_depth": depth, "seed": s["seed"] + k + 1, "estimator": 1})
        ctx.render_many(items)
        return [i[k] for i in items for k in ("pixels", "sample_count", "variance")]
    if kind == "denoise":
        ctx.atrous_device(*[v.data_ptr() for v in s["inputs"]], case["width"], case["height"], s["out"].data_ptr(),
                          stream)
        return s["out"]
    if kind == "infer":
        s["cache"].infer_device(s["queries"].data_ptr(), case["n"], s["rgb"].data_ptr(), stream)
        return s["rgb"]
    if kind == "train":
        s["cache"].train_device(s["queries"].data_ptr(), s["targets"].data_ptr(), case["n"], stream=stream)
        mlp, grid = s["grads"]
        torch.cuda.current_stream().synchronize()   # the gradients are fetched on the context's own stream
        ctx.check(ctx.lib.pico_gpu_nrc_gradients(s["cache"].handle, mlp.data_ptr(), grid.data_ptr()), "gradients")
        return [mlp, grid]
    # the file image, in a buffer of the documented bound, and its length
    ctx.check(ctx.lib.pico_gpu_encode_hdr(ctx.handle, s["image"].ctypes.data_as(ctypes.POINTER(ctypes.c_float)),
                                          case["width"], case["height"], s["file"].ctypes.data, len(s["file"]),
                                          ctypes.byref(s["length"])), "encode_hdr")
    return [s["file"], s["length"].value]


# ------------------------------------------------------------------------------- work
def _ray_flops(triangles):
    """One ray: two child boxes (25 operations each) on each level of a binary tree over the triangles, two
    triangle tests."""
    return 50.0 * math.log2(max(2, triangles)) + 100.0


def work(case):
    kind = case["kind"]
    if kind == "trace":
        return {"bytes": 52.0 * case["n"], "flops": case["n"] * _ray_flops(case["instances"] * 20 * 4 ** case["level"])}
    if kind in ("render", "cache"):
        # every pixel's image state in and out; six samples at least, one segment and one shading each
        px = case["width"] * case["height"]
        tris = {"cornell": 34, "glossy": case["instances"] * 320}.get(case.get("scene"), case["instances"] * 5120)
        return {"bytes": 56.0 * px, "flops": px * min(case["spp"], 6) * (_ray_flops(tris) + 200.0)}
    if kind == "batch":
        b = _batch(case)
        return {"bytes": sum(56.0 * w * h for w, h, *_ in b),
                "flops": sum(w * h * spp * (_ray_flops(i * 1280) + 200.0) for w, h, spp, _, i in b)}
    if kind == "denoise":
        px = case["width"] * case["height"]
        return {"bytes": 60.0 * px, "flops": 5.0 * 25.0 * 33.0 * px}
    mac = 5 * 64 * 64 + 64 * 3
    if kind == "infer":
        return {"bytes": 76.0 * case["n"] + 64.0 * (1 << case["log2_table"]), "flops": case["n"] * (2.0 * mac + 16 * 8 * 4)}
    if kind == "train":
        grid = 32.0 * (1 << case["log2_table"])
        # table read; gradient written and fetched; master, two moments read and written, table written
        return {"bytes": 80.0 * case["n"] + grid * (2 + 8 + 24 + 2), "flops": case["n"] * (6.0 * mac + 16 * 8 * 8)}
    return {"bytes": 16.0 * case["width"] * case["height"], "flops": 10.0 * case["width"] * case["height"]}


# ------------------------------------------------------------------------------- 64-bit values
def exact(case, seed):
    kind = case["kind"]
    if kind == "trace":
        tris = case["instances"] * 20 * 4 ** case["level"]
        if case["n"] * tris > 4e9:
            return None
        scene = scenes.instance_field(n_instances=case["instances"], level=case["level"], seed=seed % 100000 + 1)
        t, u, v = _exact_trace(scene, _rays(scene, case["n"], seed))
        return [None, None, t, u, v]
    if kind == "denoise":
        return _exact_atrous(*[v.double() for v in _frame(case, seed)])
    if kind in ("infer", "train"):
        q, target = _queries(case["n"], seed)
        mlp, grid = [p.double() for p in _network(case, seed)]
        if kind == "infer":
            return _exact_radiance(case, q, mlp, grid)
        mlp.requires_grad_(True)
        grid.requires_grad_(True)
        for a in range(0, case["n"], 1 << 14):
            y = _exact_radiance(case, q[a:a + (1 << 14)], mlp, grid)
            t = target[a:a + (1 << 14), :3].double()
            ((y - t) ** 2 / (y.detach() ** 2 + 0.01)).sum().div(3.0 * case["n"]).backward()
        return [mlp.grad, grid.grad]
    return None   # renders (millions of random paths) and bytes


def _exact_trace(scene, rays):
    """World distance and barycentrics of each ray's nearest triangle, by testing all of them."""
    o, d = rays[:, :3].double(), rays[:, 4:7].double()
    mesh = scene.meshes[0]
    tri = torch.from_numpy(mesh.positions.astype(np.float64)).cuda()[torch.from_numpy(mesh.indices.astype(np.int64)).cuda()]
    a, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    best = torch.full_like(o[:, 0], math.inf)
    bu, bv = torch.zeros_like(best), torch.zeros_like(best)
    rows = max(1, int(2e7 / len(a)))
    for inst in scene.instances:
        m = torch.from_numpy(np.asarray(inst.transform, np.float64).reshape(4, 4).T.copy()).cuda()
        inv = torch.linalg.inv(m)
        for r in range(0, len(o), rows):
            ro = (o[r:r + rows] @ inv[:3, :3].T + inv[:3, 3])[:, None]
            rd = (d[r:r + rows] @ inv[:3, :3].T)[:, None]
            p = torch.linalg.cross(rd, e2[None].expand(len(ro), -1, -1))
            det = (e1 * p).sum(-1)
            s = ro - a
            q = torch.linalg.cross(s, e1[None].expand(len(ro), -1, -1))
            u, v, t = (s * p).sum(-1) / det, (rd * q).sum(-1) / det, (e2 * q).sum(-1) / det
            ok = (u >= 0) & (v >= 0) & (u + v <= 1) & (t > 1e-7) & (det.abs() > 1e-7)
            t, k = torch.where(ok, t, math.inf).min(1)
            w = t * d[r:r + rows].norm(dim=1)
            nearer = w < best[r:r + rows]
            pick = torch.arange(len(k), device="cuda"), k
            bu[r:r + rows] = torch.where(nearer, u[pick], bu[r:r + rows])
            bv[r:r + rows] = torch.where(nearer, v[pick], bv[r:r + rows])
            best[r:r + rows] = torch.where(nearer, w, best[r:r + rows])
    return best, bu, bv


_KERNEL = [0.00292, 0.01306, 0.02154, 0.01306, 0.00292, 0.01306, 0.05855, 0.09653, 0.05855, 0.01306,
           0.02154, 0.09653, 0.15915, 0.09653, 0.02154, 0.01306, 0.05855, 0.09563, 0.05855, 0.01306,
           0.00292, 0.01306, 0.02154, 0.01306, 0.00292]


def _exact_atrous(pix, nrm, pos, alb):
    """Five levels of the 5x5 stencil, spacings 1 to 16; a 64x64 tile's white point and position range are over
    the pixels that its taps reach."""
    h, w, _ = pix.shape
    ys, xs = torch.arange(h, device="cuda"), torch.arange(w, device="cuda")
    length = pos.norm(dim=2)
    weights = [float(np.float32(k)) for k in _KERNEL]
    lum = torch.tensor([float(np.float32(v)) for v in (0.2126, 0.587, 0.114)], dtype=torch.float64, device="cuda")
    for level in range(5):
        s = 1 << level
        taps = [(ys + (j - 2) * s).clamp(0, h - 1) for j in range(5)], [(xs + (i - 2) * s).clamp(0, w - 1) for i in range(5)]
        white, reach = torch.empty_like(length), torch.empty_like(length)
        bright = pix @ lum
        for y0 in range(0, h, 64):
            rows = torch.unique(torch.cat([t[y0:y0 + 64] for t in taps[0]]))
            for x0 in range(0, w, 64):
                cols = torch.unique(torch.cat([t[x0:x0 + 64] for t in taps[1]]))
                b = bright[rows][:, cols]
                white[y0:y0 + 64, x0:x0 + 64] = torch.where(b.isnan(), 0.0, b).amax().clamp_min(0.0)
                l = length[rows][:, cols]
                reach[y0:y0 + 64, x0:x0 + 64] = l.amax() - l.amin()
        total, norm = torch.zeros_like(pix), torch.zeros_like(length)
        for j in range(5):
            for i in range(5):
                at = (taps[0][j][:, None], taps[1][i][None, :])
                wn = torch.exp(-((nrm - nrm[at]) ** 2).sum(2) / 0.25)
                wp = torch.exp(-((pos - pos[at]) ** 2).sum(2) / reach ** 2)
                wa = torch.exp(-((alb - alb[at]) ** 2).sum(2) / white ** 2)
                k = weights[j * 5 + i] * wn * wp * wa
                total += k[:, :, None] * pix[at]
                norm += k
        pix = total / norm[:, :, None]
    return pix


def _exact_radiance(case, q, mlp, grid):
    """The cache's network on query records: hash grid, spherical harmonics, five hidden layers."""
    q = q.double()
    lo, hi = (torch.tensor(b, dtype=torch.float64, device="cuda") for b in BOUNDS)
    u = ((q[:, 0:3] - lo) / (hi - lo)).clamp(0.0, 1.0)
    size = 1 << case["log2_table"]
    feats = []
    for level in range(16):
        scale = 16.0 * (4096.0 / 16.0) ** (level / 15.0)
        side = int(math.floor(float(np.float32(scale)))) + 2
        x = u * scale
        c = x.floor()
        f = x - c
        c = c.long()
        total = 0.0
        for k in range(8):
            bits = torch.tensor([k & 1, k >> 1 & 1, k >> 2], device="cuda")
            p = c + bits
            if side ** 3 <= size:
                at = p[:, 0] + side * (p[:, 1] + side * p[:, 2])
            else:
                at = (p[:, 0] ^ (p[:, 1] * 2654435761 & 0xffffffff) ^ (p[:, 2] * 805459861 & 0xffffffff)) & (size - 1)
            wt = torch.where(bits == 1, f, 1.0 - f).prod(1)
            total = total + wt[:, None] * grid[level][at]
        feats.append(total)
    x, y, z = q[:, 3], q[:, 4], q[:, 5]
    xx, yy, zz = x * x, y * y, z * z
    r = lambda v: math.sqrt(v / math.pi)   # noqa: E731
    sh = [0.5 * r(1) + 0 * x, -r(3 / 4) * y, r(3 / 4) * z, -r(3 / 4) * x, r(15 / 4) * x * y, -r(15 / 4) * y * z,
          r(5 / 16) * (3 * zz - 1), -r(15 / 4) * x * z, r(15 / 16) * (xx - yy), -r(35 / 32) * y * (3 * xx - yy),
          r(105 / 4) * x * y * z, -r(21 / 32) * y * (5 * zz - 1), r(7 / 16) * z * (5 * zz - 3),
          -r(21 / 32) * x * (5 * zz - 1), r(105 / 16) * z * (xx - yy), -r(35 / 32) * x * (xx - 3 * yy)]
    v = torch.cat(feats + [torch.stack(sh, 1), q[:, 6:13], torch.ones_like(x)[:, None],
                           torch.zeros(len(q), 8, dtype=torch.float64, device="cuda")], 1)
    for l in range(5):
        v = torch.relu(v @ mlp[l].T)
    return (v @ mlp[5].T)[:, :3]
