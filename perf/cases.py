"""The workloads by which this renderer's speed is followed.

Each case is one pass through a public entry point of `alpine_b200.gpu`: batched
ray queries, BVH (re)builds, renders, and the learned guide's inference and
gradients. `listed()` names the fixed ones, `draw()` gives more of the same
ranges, `prepare()` makes what a program holds before the call, `run()` is one
pass, `work()` its unavoidable bytes and operations, and `exact()` its outputs
in 64 bits where they are computed numbers with a closed form.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from alpine_b200 import batch, gpu, scenes

FLT_MAX = 3.4028234663852886e38
GUIDE_LO, GUIDE_HI = (-1.0, -1.0, -1.0), (1.0, 1.0, 1.0)
GUIDE_RES = (16, 32, 64, 128, 256, 512, 1024, 2048)
GUIDE_TABLE, GUIDE_FEATURES = 1 << 19, 4
GUIDE_LAYERS = ((64, 64), (64, 64), (64, 64), (64, 64), (48, 64))  # (out, in)


def listed():
    return [
        # one 16 x 16 image tile handed to the accelerator from host memory: the smallest
        # call, all latency
        {"name": "query_tile_host", "kind": "query", "scene": "room", "tris": 4036, "rays": 256, "coherent": 1.0,
         "any": False, "rule": "wide", "via": "pageable"},
        # the traversal benchmark's closest-hit half: a million-triangle soup, primary rays
        # then incoherent ones, on the device
        {"name": "query_closest_4m", "kind": "query", "scene": "soup", "tris": 1 << 20, "rays": 1 << 22,
         "coherent": 0.5, "any": False, "rule": "wide", "via": "device"},
        # shadow rays of an integrator: any hit, odd sizes, the binary accelerator's triangle rule
        {"name": "query_shadow_ragged", "kind": "query", "scene": "soup", "tris": 300_007, "rays": 1_000_003,
         "coherent": 0.0, "any": True, "rule": "binary", "via": "device"},
        # a batch from pinned host memory and back, as a CPU renderer uses the accelerator
        {"name": "query_pinned_1m", "kind": "query", "scene": "soup", "tris": 1 << 20, "rays": 1 << 20,
         "coherent": 0.5, "any": False, "rule": "wide", "via": "pinned"},
        # a large static scene: the first build, and the first image's primary rays through it
        {"name": "build_soup_1m", "kind": "rebuild", "scene": "soup", "tris": 1 << 20, "rays": 131_072,
         "driver": "static"},
        # a small animated scene: morph, host-driven rebuild, primary rays
        {"name": "animate_host_8k", "kind": "rebuild", "scene": "batch", "tris": 8_000, "rays": 16_384,
         "driver": "host"},
        # a frame of the animated batch: morph, device-driven rebuild and render with nothing
        # waited for in between, then the image
        {"name": "frame_batch_60k", "kind": "render", "scene": "batch", "tris": 60_000, "width": 256, "height": 256,
         "spp": 4, "depth": 8, "sampler": "bvh", "roulette": 3, "animate": True, "graph": True, "guide": False,
         "fp64": False},
        # the small room with next-event estimation
        {"name": "render_room", "kind": "render", "scene": "room", "tris": 4036, "width": 256, "height": 256,
         "spp": 16, "depth": 8, "sampler": "power", "roulette": 3, "animate": False, "graph": False, "guide": False,
         "fp64": False},
        # a city lit by many windows, light-BVH sampling
        {"name": "render_city", "kind": "render", "scene": "city", "tris": 240_000, "width": 960, "height": 540,
         "spp": 2, "depth": 8, "sampler": "bvh", "roulette": 0, "animate": False, "graph": False, "guide": False,
         "fp64": False},
        # the glossy interior of two million triangles, with a guide that has stopped training
        {"name": "render_interior_guided", "kind": "render", "scene": "interior", "tris": 2_000_000, "width": 640,
         "height": 360, "spp": 8, "depth": 12, "sampler": "none", "roulette": 0, "animate": False, "graph": False,
         "guide": True, "fp64": True},
        # the guide alone: one bounce's queries of a large wave
        {"name": "guide_infer_1m", "kind": "infer", "n": (1 << 20) + 1, "kernel": "warp_mma"},
        # the guide's backward pass over one training batch
        {"name": "guide_gradients_16k", "kind": "gradients", "n": 16_384},
    ]


def _log_int(rng, lo, hi):
    return int(math.exp(rng.uniform(math.log(lo), math.log(hi))))


def draw(rng):
    kind = rng.choice(("query", "query", "query", "rebuild", "rebuild", "render", "render", "infer", "gradients"))
    if kind == "query":
        scene = rng.choice(("room", "soup", "soup"))
        return {"kind": kind, "scene": scene, "tris": 4036 if scene == "room" else _log_int(rng, 1_000, 1_000_000),
                "rays": _log_int(rng, 200, 2_000_000),
                "coherent": 1.0 if scene == "room" else rng.choice((0.0, 0.5, 1.0)), "any": rng.random() < 0.4,
                "rule": rng.choice(("wide", "wide", "binary")), "via": rng.choice(("device", "device", "pinned", "pageable"))}
    if kind == "rebuild":
        scene = rng.choice(("soup", "batch", "batch"))
        return {"kind": kind, "scene": scene, "tris": _log_int(rng, 1_000, 1_000_000 if scene == "soup" else 300_000),
                "rays": _log_int(rng, 1_000, 131_072),
                "driver": "static" if scene == "soup" else rng.choice(("host", "device"))}
    if kind == "render":
        scene = rng.choice(("room", "batch", "interior"))
        w, h = _log_int(rng, 64, 512), _log_int(rng, 64, 512)
        spp = max(1, min(16, _log_int(rng, 65_536, 1_000_000) // (w * h)))
        guide = scene == "interior" and rng.random() < 0.7
        return {"kind": kind, "scene": scene, "tris": 4036 if scene == "room" else _log_int(rng, 2_000, 300_000),
                "width": w, "height": h, "spp": spp, "depth": rng.choice((4, 8, 12)),
                "sampler": "none" if scene == "interior" else rng.choice(("uniform", "power", "bvh")),
                "roulette": rng.choice((0, 3)), "animate": scene == "batch" and rng.random() < 0.6,
                "graph": scene != "interior" and rng.random() < 0.5, "guide": guide, "fp64": rng.random() < 0.3}
    if kind == "infer":
        return {"kind": kind, "n": _log_int(rng, 100, 1_000_000), "kernel": rng.choice(("warp_mma", "tensor_memory"))}
    return {"kind": kind, "n": _log_int(rng, 100, 65_536)}


# ---------------------------------------------------------------------------
# inputs
def _generator(seed, salt):
    g = torch.Generator(device="cuda")
    g.manual_seed(1_000_003 * int(seed) + salt)
    return g


def _unit(g, n):
    v = torch.randn(n, 3, generator=g, device="cuda", dtype=torch.float64)
    return v / v.norm(dim=1, keepdim=True)


def _scene(case, seed):
    """A scene description (alpine_b200/scenes.py) of about case["tris"] triangles."""
    if case["scene"] == "room":
        return scenes.room_scene(seed=seed, light="quad")
    if case["scene"] == "city":
        # about 600 triangles and 50 windows a building
        n = max(1, case["tris"] // 600)
        return scenes.city_scene(seed=seed, buildings=n, lights=50 * n, extent=max(200.0, 50.0 * math.sqrt(n)))
    if case["scene"] == "interior":
        return scenes.glossy_interior_scene(seed=seed, target_tris=case["tris"])
    if case["scene"] == "batch":
        return batch.batch_scene(seed, case["tris"])
    verts, idx = scenes.triangle_soup(case["tris"], seed=seed)
    camera = ((0.5, 0.5, -1.0), (0.5, 0.5, 0.0), (0.0, 1.0, 0.0), math.radians(60.0))
    return {"meshes": [{"verts": verts, "idx": idx, "normals": None, "tri_material": np.zeros(idx.shape[0], np.uint32)}],
            "materials": [(0, (0.5, 0.5, 0.5), 1.0)], "lights": [], "camera": camera, "background": (0.0, 0.0, 0.0)}


def _camera_rays(camera, n, g):
    """n rays of a 2:1 image through jittered pixel positions, row by row, from `camera`."""
    eye, target, up, fovy = camera
    x, y, z = (torch.from_numpy(a).cuda() for a in scenes.look_at_basis(eye, target, up))
    w = max(1, int(math.ceil(math.sqrt(2.0 * n))))
    h = -(-n // w)
    i = torch.arange(n, device="cuda")
    jitter = torch.rand(n, 2, generator=g, device="cuda", dtype=torch.float64)
    fh = math.tan(0.5 * fovy)
    fx = ((i % w + jitter[:, 0]) / w - 0.5) * (2.0 * fh)
    fy = (0.5 - (i // w + jitter[:, 1]) / h) * fh
    d = fx[:, None] * x + fy[:, None] * y + z
    o = torch.tensor(eye, device="cuda", dtype=torch.float64).expand(n, 3)
    return o, d / d.norm(dim=1, keepdim=True)


def _rays(case, camera, seed):
    """float32 [n, 8] rays on the GPU: camera rays, then rays of random origins in the unit
    cube and random directions; any-hit rays have tmax uniform in (0, 1]."""
    n, g = case["rays"], _generator(seed, 1)
    nc = int(round(n * case.get("coherent", 1.0)))
    o1, d1 = _camera_rays(camera, nc, g)
    o2 = torch.rand(n - nc, 3, generator=g, device="cuda", dtype=torch.float64)
    d2 = _unit(g, n - nc)
    rays = torch.zeros(n, 8, device="cuda", dtype=torch.float32)
    rays[:, 0:3] = torch.cat([o1, o2]).float()
    rays[:, 4:7] = torch.cat([d1, d2]).float()
    rays[:, 7] = 1.0 - torch.rand(n, generator=g, device="cuda") if case.get("any") else FLT_MAX
    return rays


def _guide_parameters(seed):
    """Weights (packed layer after layer, [out][in]; the output layer's a quarter as large, for
    lobes of moderate width) and the whole hash grid, float32 on the GPU."""
    g = _generator(seed, 2)
    w = torch.cat([(2.0 * torch.rand(o * i, generator=g, device="cuda") - 1.0) * math.sqrt(6.0 / i) *
                   (0.25 if l == len(GUIDE_LAYERS) - 1 else 1.0) for l, (o, i) in enumerate(GUIDE_LAYERS)])
    grid = torch.rand(len(GUIDE_RES) * GUIDE_TABLE * GUIDE_FEATURES, generator=g, device="cuda") - 0.5
    return w, grid


def _guide_queries(n, seed):
    """float32 [n, 12]: position, roughness, direction, 0, normal, 0."""
    g = _generator(seed, 3)
    q = torch.zeros(n, 12, device="cuda", dtype=torch.float32)
    q[:, 0:3] = 2.0 * torch.rand(n, 3, generator=g, device="cuda") - 1.0
    q[:, 3] = 0.02 + 0.98 * torch.rand(n, generator=g, device="cuda")
    q[:, 4:7] = _unit(g, n).float()
    q[:, 8:11] = _unit(g, n).float()
    return q


def _guide_samples(n, seed):
    """float32 [n, 16]: a query, a sampled direction and the weight of its gradient."""
    g = _generator(seed, 4)
    s = torch.zeros(n, 16, device="cuda", dtype=torch.float32)
    s[:, 0:12] = _guide_queries(n, seed)
    s[:, 12:15] = _unit(g, n).float()
    s[:, 15] = torch.exp(torch.randn(n, generator=g, device="cuda"))
    return s


def _grid_index(seed):
    """The grid parameters whose gradients are asked for: the coarsest level's, and some of the others."""
    first = np.arange((GUIDE_RES[0] + 1) ** 3 * GUIDE_FEATURES, dtype=np.uint64)
    rest = np.random.default_rng(seed).integers(0, len(GUIDE_RES) * GUIDE_TABLE * GUIDE_FEATURES, 32_768)
    return np.concatenate([first, rest.astype(np.uint64)])


def _load_guide(ctx, seed, lo=GUIDE_LO, hi=GUIDE_HI):
    """Sets the guide's parameters, positions normalised to the box [lo, hi]."""
    w, grid = _guide_parameters(seed)
    ctx.guide_reset(seed % (1 << 31), lo, hi)
    ctx.guide_set_weights(w.cpu().numpy())
    ctx.guide_grid(np.arange(grid.numel(), dtype=np.uint64), write=grid.cpu().numpy())


# ---------------------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "time": float(seed % batch.FRAMES) + 0.25}
    if kind in ("query", "rebuild"):
        scene = _scene(case, seed)
        c = s["ctx"] = gpu.Context(0)
        scenes.load_scene(c, scene, 2, 1)
        if case.get("rule") == "binary":
            c.set_traversal_options(triangle_test=gpu.TRIANGLE_TEST_BINARY_BVH)
        rays = _rays(case, scene["camera"], seed)
        n = case["rays"]
        out = torch.empty(n, dtype=torch.uint8) if case.get("any") else torch.empty(n, 4, dtype=torch.int32)
        via = case.get("via", "device")
        if via == "device":
            s["rays"], out = rays, out.cuda()
        else:
            rays = rays.cpu()
            s["rays"], out = (rays.pin_memory(), out.pin_memory()) if via == "pinned" else (rays, out)
            s["rays_host"], s["out_host"] = s["rays"].numpy(), out.numpy()
        s["out"] = out
        # the hit records' fields, as the caller reads them
        s["fields"] = {"occluded": out} if case.get("any") else {
            "prim": out[:, 0], "t": out[:, 1].view(torch.float32), "b1": out[:, 2].view(torch.float32),
            "b2": out[:, 3].view(torch.float32)}
    elif kind == "render":
        c = s["ctx"] = gpu.Context(0, case["width"], case["height"], case["depth"])
        scenes.load_scene(c, _scene(case, seed), case["width"], case["height"])
        if case["sampler"] != "none":
            c.build_light_sampler({"uniform": gpu.SAMPLER_UNIFORM, "power": gpu.SAMPLER_POWER,
                                   "bvh": gpu.SAMPLER_BVH}[case["sampler"]])
        if case["guide"]:
            _load_guide(c, seed, (-10.0, 0.0, -6.0), (10.0, 4.0, 6.0))
        c.set_render_options(sampler=gpu.RNG_COUNTER, seed=seed % (1 << 31), russian_roulette_depth=case["roulette"],
                             accumulate_fp64=case["fp64"], cuda_graph=case["graph"], guide=case["guide"],
                             guide_train=False, guide_min_roughness=0.2)
    else:
        c = s["ctx"] = gpu.Context(0)
        _load_guide(c, seed)
        if kind == "infer":
            c.guide_set_kernel(gpu.GUIDE_KERNEL_TENSOR_MEMORY if case["kernel"] == "tensor_memory"
                               else gpu.GUIDE_KERNEL_WARP_MMA)
            s["queries"] = _guide_queries(case["n"], seed)
            s["raw"] = torch.empty(case["n"], 40, device="cuda", dtype=torch.float32)
        else:
            s["samples"] = _guide_samples(case["n"], seed).cpu().numpy()
            s["index"] = _grid_index(seed)
    return s


def run(s):
    case, c = s["case"], s["ctx"]
    kind = case["kind"]
    if kind == "query":
        via = case["via"]
        if via == "device":
            (c.occluded_device if case["any"] else c.trace_device)(s["rays"].data_ptr(), case["rays"],
                                                                   s["out"].data_ptr())
        else:
            (c.occluded if case["any"] else c.trace)(s["rays_host"], out=s["out_host"])
        return s["fields"]
    if kind == "rebuild":
        if case["driver"] == "static":
            c.build()
        elif case["driver"] == "host":
            c.update_scene(s["time"])
        else:
            c.update_scene_async(s["time"])
        c.trace_device(s["rays"].data_ptr(), case["rays"], s["out"].data_ptr())
        return s["fields"]
    if kind == "render":
        c.reset_accumulation()
        if case["animate"]:
            c.update_scene_async(s["time"])
            c.render_async(case["spp"])
            c.render_wait()
        else:
            c.render(case["spp"])
        sums, samples = c.read_accumulation(case["width"], case["height"], fp64=case["fp64"])
        return {"sums": sums, "samples": samples}
    if kind == "infer":
        c.guide_infer_device(s["queries"].data_ptr(), case["n"], s["raw"].data_ptr())
        return s["raw"]
    weights, grid = c.guide_gradients(s["samples"], s["index"])
    return {"weights": weights, "grid": grid}


def work(case):
    kind = case["kind"]
    if kind in ("query", "rebuild"):
        n, t = case["rays"], case["tris"]
        out = 1 if case.get("any") else 16
        # a ray meets about one 8-wide node (8 boxes, 12 operations each) per halving of the
        # triangle count, and four triangles (50 operations)
        flops = n * (96.0 * math.log2(t) + 200.0)
        size = n * (32.0 + out) + 48.0 * min(t, 4 * n)
        if kind == "rebuild":  # vertices and indices in, triangle records and nodes out; binning per level
            size += t * (48.0 + 48.0 + 14.0)
            flops += t * math.log2(t) * 30.0
        return {"bytes": size, "flops": flops}
    if kind == "render":
        paths = case["width"] * case["height"] * case["spp"]
        size = case["width"] * case["height"] * 9.0 * (8 if case["fp64"] else 4) + 64.0 * case["tris"]
        vertex = 96.0 * math.log2(case["tris"]) + 600.0 + (40_000.0 if case["guide"] else 0.0)
        mean_depth = min(case["depth"], 4.0) if case["roulette"] else 0.7 * case["depth"]
        return {"bytes": size, "flops": paths * mean_depth * vertex}
    mlp = 2.0 * sum(o * i for o, i in GUIDE_LAYERS)
    if kind == "infer":
        return {"bytes": case["n"] * (48.0 + 160.0 + 8 * 8 * 8.0), "flops": case["n"] * mlp}
    # samples in, the gradients of the touched grid entries and of the weights out
    return {"bytes": case["n"] * (64.0 + 2 * 8 * 8 * 16.0), "flops": 3.0 * case["n"] * mlp}


# ---------------------------------------------------------------------------
# 64-bit outputs
def _closest_exact(case, seed):
    """Closest hits by testing every triangle (t, b1, b2; FLT_MAX, 0, 0 for a miss)."""
    scene = _scene(case, seed)
    rays = _rays(case, scene["camera"], seed).double()
    tri = np.concatenate([np.asarray(m["verts"], np.float32)[m["idx"]] for m in scene["meshes"]])
    tri = torch.from_numpy(tri).cuda().double()
    v0, e0, e1 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    out = torch.empty(rays.shape[0], 3, dtype=torch.float64, device="cuda")
    step = max(1, 4_000_000 // tri.shape[0])
    for a in range(0, rays.shape[0], step):
        o, d = rays[a:a + step, None, 0:3], rays[a:a + step, None, 4:7]
        sv = o - v0
        s1 = torch.linalg.cross(d.expand(-1, tri.shape[0], 3), e1.expand(d.shape[0], -1, 3))
        s2 = torch.linalg.cross(sv, e0.expand(d.shape[0], -1, 3))
        det = (s1 * e0).sum(-1)
        b1, b2, t = (s1 * sv).sum(-1) / det, (d * s2).sum(-1) / det, (s2 * e1).sum(-1) / det
        ok = (det.abs() >= 1e-6) & (t >= 0) & (b1 >= 0) & (b2 >= 0) & (b1 + b2 <= 1)
        t = torch.where(ok, t, torch.inf)
        k = t.argmin(1, keepdim=True)
        hit = torch.isfinite(t.gather(1, k))[:, 0]
        r = torch.stack([t.gather(1, k)[:, 0], b1.gather(1, k)[:, 0], b2.gather(1, k)[:, 0]], 1)
        miss = torch.tensor([FLT_MAX, 0.0, 0.0], dtype=torch.float64, device="cuda")
        out[a:a + step] = torch.where(hit[:, None], r, miss)
    return {"prim": None, "t": out[:, 0], "b1": out[:, 1], "b2": out[:, 2]}


def _rounded(x, dtype):
    """x as `dtype` holds it, in 64 bits; its derivative is x's own."""
    return x + (x.detach().to(dtype).double() - x.detach())


def _guide_forward(w, grid, q, stored=False):
    """The 40 mixture parameters of every query, in 64 bits (differentiable). stored: from the
    parameters and layer inputs as the model holds them in 16 bits, which decide the ReLU
    masks of its backward pass."""
    if stored:
        w, grid = _rounded(w, torch.bfloat16), _rounded(grid, torch.float16)
    lo = torch.tensor(GUIDE_LO, dtype=torch.float64, device="cuda")
    extent = (max(h - l for h, l in zip(GUIDE_HI, GUIDE_LO))) * 1.0001
    p = ((q[:, 0:3].double() - lo) / extent).clamp(0.0, 0.99999)
    feats = []
    for l, res in enumerate(GUIDE_RES):
        f = p * res
        i = f.floor()
        t, i = f - i, i.long()
        acc = 0.0
        for c in range(8):
            o = [c & 1, (c >> 1) & 1, (c >> 2) & 1]
            x, y, z = (i[:, k] + o[k] for k in range(3))
            if (res + 1) ** 3 <= GUIDE_TABLE:
                e = x + (res + 1) * (y + (res + 1) * z)
            else:
                e = (x ^ (y * 2654435761) ^ (z * 805459861)) & (GUIDE_TABLE - 1)
            wt = 1.0
            for k in range(3):
                wt = wt * (t[:, k] if o[k] else 1.0 - t[:, k])
            acc = acc + wt[:, None] * grid[l * GUIDE_TABLE + e]
        feats.append(acc)
    n = q[:, 8:11].double()
    h = torch.cat(feats + [q[:, 4:7].double(), n / n.norm(dim=1, keepdim=True), q[:, 3:4].double(),
                           torch.ones_like(q[:, 3:4], dtype=torch.float64),
                           torch.zeros(q.shape[0], 24, dtype=torch.float64, device="cuda")], 1)
    at = 0
    for l, (o, i) in enumerate(GUIDE_LAYERS):
        h = (_rounded(h, torch.bfloat16) if stored else h) @ w[at:at + o * i].view(o, i).T
        at += o * i
        if l < len(GUIDE_LAYERS) - 1:
            h = h.relu()
    return h[:, :40]


def _guide_gradients_exact(n, seed):
    w, grid = _guide_parameters(seed)
    w = w.double().requires_grad_()
    grid = grid.double().view(-1, GUIDE_FEATURES).requires_grad_()
    s = _guide_samples(n, seed)
    r = _guide_forward(w, grid, s[:, 0:12], stored=True).view(n, 8, 5)
    mu = r[..., 0:3] / r[..., 0:3].norm(dim=-1, keepdim=True)
    kappa = r[..., 3].clamp(-2.0, 8.0).exp()
    v = kappa / (2.0 * math.pi * -torch.expm1(-2.0 * kappa)) * torch.exp(
        kappa * ((mu * s[:, None, 12:15].double()).sum(-1) - 1.0))
    pdf = (torch.softmax(r[..., 4], -1) * v).sum(-1)
    (-(s[:, 15].double() * pdf.clamp_min(1e-30).log()).sum() / n).backward()
    return {"weights": w.grad, "grid": grid.grad.view(-1)[torch.from_numpy(_grid_index(seed).astype(np.int64)).cuda()]}


def exact(case, seed):
    kind = case["kind"]
    if kind == "query" and case["scene"] == "room" and not case["any"] and case["rays"] * case["tris"] <= 200_000_000:
        return _closest_exact(case, seed)
    if kind == "infer":
        w, grid = _guide_parameters(seed)
        return _guide_forward(w.double(), grid.double().view(-1, GUIDE_FEATURES), _guide_queries(case["n"], seed))
    if kind == "gradients":
        return _guide_gradients_exact(case["n"], seed)
    return None
