"""The work that users of yar_gb300 have it do, as cases whose time is measured.

Each case goes through the package's public entry points (`native.Context`): ray casts over batches in host and
device memory, the path tracer, the direct-lighting renderer, the batched render, the guided render and the guide
network.  A state keeps what a program keeps between calls: the context with its uploaded scene, the rays, the
network's rows.  The geometry of a case is fixed; the seed gives the rays, the pixels' sample streams, the network's
weights and rows.
"""
import functools
import math
import os

import numpy as np
import torch

from yar_gb300 import native, scenes
from yar_gb300.scene import FlatScene

GOLDEN = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "tests", "golden")
BOX = (-1.0, 0.0, -1.0, 1.0, 2.0, 1.0)  # scene bounds of the guide network's positions


def listed():
    return [
        # a viewport's picking and probing: a thousand rays from host memory, latency counts
        dict(name="cast-closest-host-1k", kind="cast", ray="closest", buffers="host", grid=128, spheres=8, rays=1021),
        # a simulation step of a host program: an odd million of rays, copies inside the call
        dict(name="cast-closest-host-1m", kind="cast", ray="closest", buffers="host", grid=512, spheres=64,
             rays=1000003),
        # the ray-cast benchmark (2.42M triangles, 16M incoherent rays in device memory), closest hit and shadow rays
        dict(name="cast-closest-16m", kind="cast", ray="closest", buffers="device", grid=1024, spheres=64,
             rays=16777216),
        dict(name="cast-any-16m", kind="cast", ray="any", buffers="device", grid=1024, spheres=64, rays=16777216),
        # a small preview render: the diffuse Cornell box, 256 x 256 at 16 samples, depth 8
        dict(name="render-cornell-256", kind="render", scene="cornell_c1_64", width=256, height=256, side=4, depth=8),
        # a final frame: 4.1M triangles, GGX and diffuse, 64 lights, 1080p, depth 16
        dict(name="render-large-1080p", kind="render", scene="large", width=1920, height=1080, side=4, depth=16),
        # indirect light only: the closed GGX room of 480K triangles
        dict(name="render-room-512", kind="render", scene="room", width=512, height=512, side=8, depth=12),
        # image textures, bump maps, mirror and smooth glass: the full shading code, an odd image size
        dict(name="render-textured-333", kind="render", scene="cornell_spectex_64", width=333, height=251, side=4,
             depth=8),
        # the direct-lighting algorithm with quad, point, spot and distant lights
        dict(name="render-direct-512", kind="render", scene="cornell_direct_64", width=512, height=512, side=4,
             depth=8),
        # six scenes of uneven size in one call
        dict(name="render-batch-6", kind="batch", scenes=6, first=4),
        # the room with continuations drawn from a kept proposal
        dict(name="guided-room-512", kind="guided", width=512, height=512, spp=64, depth=12),
        # a training loop of one's own over the proposal: its loss gradient, then its mixtures at new points
        dict(name="guide-network", kind="network", infer_rows=1048576, train_rows=262144),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["cast", "cast", "cast", "render", "render", "render", "network", "guided", "batch"])
    if kind == "cast":
        buffers = rng.choice(["host", "device"])
        return dict(kind=kind, ray=rng.choice(["closest", "any"]), buffers=buffers, grid=_log_int(rng, 32, 700),
                    spheres=rng.randint(0, 64), rays=_log_int(rng, 1, 2000000 if buffers == "host" else 16777216))
    if kind == "render":
        scene = rng.choice(["cornell_c1_64", "cornell_ggx_64", "cornell_spectex_64", "cornell_bump_64",
                            "cornell_direct_64", "cornell_lights_64", "room", "medium"])
        return dict(kind=kind, scene=scene, width=_log_int(rng, 48, 700), height=_log_int(rng, 48, 500),
                    side=rng.randint(1, 5), depth=rng.randint(2, 14))
    if kind == "network":
        return dict(kind=kind, infer_rows=_log_int(rng, 1, 1048576), train_rows=_log_int(rng, 16, 262144))
    if kind == "guided":
        return dict(kind=kind, width=_log_int(rng, 64, 512), height=_log_int(rng, 64, 512), spp=rng.randint(4, 60),
                    depth=rng.randint(4, 12))
    return dict(kind=kind, scenes=rng.randint(2, 6), first=rng.randint(5, 40))


# ---------------------------------------------------------------- geometry (the same for every seed)
@functools.lru_cache(maxsize=4)
def _cast_scene(grid, spheres):
    return scenes.raycast_scene(seed=1, grid=grid, spheres=spheres, level=4 if grid >= 256 else 2)


@functools.lru_cache(maxsize=2)
def _built_scene(name):
    if name == "large":
        return scenes.large_scene(seed=1)
    if name == "medium":
        return scenes.large_scene(seed=3, meshes=40, level=4, lights=9)
    return scenes.hard_lighting_room(seed=1)


@functools.lru_cache(maxsize=2)
def _batch(first, count):
    return scenes.batch_scenes(seed=first, count=count)


def _render_scene(case, seed):
    name = case["scene"]
    s = FlatScene.read(os.path.join(GOLDEN, name + ".yfs")) if name.startswith("cornell") else _built_scene(name)
    w, h = case["width"], case["height"]
    s.camera = np.array(s.camera)
    s.config = np.array(s.config)
    s.camera["image_extent"] = (w, h)
    s.camera["horz_half_dist"] = np.float32(np.float32(w) / np.float32(h)) * np.float32(s.camera["vert_half_dist"])
    s.config["render_region"] = (0, 0, w, h)
    s.config["x_pixel_sample_count"] = s.config["y_pixel_sample_count"] = case.get("side", 1)
    s.config["max_light_bounces"] = case["depth"]
    s.config["rng_seed_offset"] = _offset(seed)
    return s


def _offset(seed):
    return 1 + (int(seed) * 7919) % (1 << 28)


# ---------------------------------------------------------------- inputs
def _unit(n, g):
    v = torch.randn((n, 3), device="cuda", generator=g)
    return v / v.norm(dim=1, keepdim=True)


def _rays(s, n, ray, seed):
    """Origins uniform in the scene box, directions uniform on the sphere; closest-hit rays reach past the box,
    shadow rays have lengths uniform up to its diagonal."""
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    lo = torch.tensor(s.scene_bounds[:3], device="cuda")
    hi = torch.tensor(s.scene_bounds[3:], device="cuda")
    diag = float((hi - lo).norm())
    rays = torch.zeros((n, 8), device="cuda")
    rays[:, 0:3] = lo + (hi - lo) * torch.rand((n, 3), device="cuda", generator=g)
    rays[:, 3] = 2.0 * diag if ray == "closest" else diag * torch.rand(n, device="cuda", generator=g)
    rays[:, 4:7] = _unit(n, g)
    return rays


def _rows(n, width, g):
    r = torch.zeros((n, width), device="cuda")
    lo = torch.tensor(BOX[:3], device="cuda")
    hi = torch.tensor(BOX[3:], device="cuda")
    r[:, 0:3] = lo + (hi - lo) * torch.rand((n, 3), device="cuda", generator=g)
    for c in (3, 6) + ((9,) if width == 16 else ()):
        r[:, c:c + 3] = _unit(n, g)
    if width == 16:
        r[:, 12] = torch.rand(n, device="cuda", generator=g)
    return r


def _network_params(seed):
    """Weights as the proposal is initialised: uniform by fan-in, the outputs small."""
    rng = np.random.default_rng([int(seed), 17])
    w1 = rng.uniform(-1, 1, (64, 128)) * math.sqrt(6 / 102)
    w2, w3, w4 = (rng.uniform(-1, 1, (64, 64)) * math.sqrt(6 / 63) for _ in range(3))
    w4 *= 0.5
    w4[40:] = 0.0
    return np.concatenate([w.ravel() for w in (w1, w2, w3, w4)]).astype(np.float32)


def prepare(case, seed):
    state = dict(case=case, ctx=native.Context(0))
    ctx, kind = state["ctx"], case["kind"]
    if kind == "cast":
        s = _cast_scene(case["grid"], case["spheres"])
        ctx.upload_scene(s)
        n = case["rays"]
        rays = _rays(s, n, case["ray"], seed)
        if case["buffers"] == "host":
            state["rays"] = rays.cpu().numpy()
        else:
            state["rays"] = rays
            if case["ray"] == "closest":
                state["out"] = [torch.empty(n, device="cuda"), torch.empty(n, dtype=torch.int32, device="cuda"),
                                torch.empty(n, dtype=torch.int32, device="cuda"), torch.empty((n, 2), device="cuda")]
            else:
                state["out"] = [torch.empty(n, dtype=torch.uint8, device="cuda")]
    elif kind == "render":
        ctx.upload_scene(_render_scene(case, seed))
    elif kind == "batch":
        state["flats"] = _batch(case["first"], case["scenes"])
        state["offset"] = _offset(seed)
    elif kind == "guided":
        ctx.upload_scene(_render_scene(dict(case, scene="room"), seed))
        ctx.guide_set_params(_network_params(seed))
        state["offset"] = 1 + int(seed) % 4000
    else:
        g = torch.Generator(device="cuda").manual_seed(int(seed))
        ctx.guide_set_params(_network_params(seed))
        state["queries"] = _rows(case["infer_rows"], 12, g)
        state["samples"] = _rows(case["train_rows"], 16, g)
        state["lobes"] = torch.empty((case["infer_rows"], native.GUIDE_LOBE_FLOATS), device="cuda")
        state["grad"] = torch.empty(native.GUIDE_PARAMS, device="cuda")
    torch.cuda.synchronize()
    return state


def run(state):
    case, ctx = state["case"], state["ctx"]
    kind = case["kind"]
    if kind == "cast":
        rays = state["rays"]
        if case["buffers"] == "host":
            return ctx.cast_closest(rays) if case["ray"] == "closest" else ctx.cast_any(rays)
        out = state["out"]
        if case["ray"] == "closest":
            ctx.cast_closest_device(rays.data_ptr(), case["rays"], *(o.data_ptr() for o in out))
        else:
            ctx.cast_any_device(rays.data_ptr(), case["rays"], out[0].data_ptr())
        return out
    if kind == "render":
        image, stats = ctx.render(case["width"], case["height"])
        return image, stats.variance
    if kind == "batch":
        for flat in state["flats"]:
            flat.config["rng_seed_offset"] = state["offset"]
        images, scene_stats, _ = ctx.render_batch(state["flats"])
        return images, [s.variance for s in scene_stats]
    if kind == "guided":
        image, sums, _ = ctx.guided_render(case["width"], case["height"], guide_fraction=0.6,
                                           samples_per_pixel=case["spp"], guide_bounces=2, keep_guide=True,
                                           stream_offset=state["offset"])
        return image, sums
    loss = ctx.guide_gradient(state["samples"].data_ptr(), case["train_rows"], BOX, 1.0 / case["train_rows"],
                              state["grad"].data_ptr())
    ctx.guide_infer(state["queries"].data_ptr(), case["infer_rows"], BOX, state["lobes"].data_ptr())
    return loss, state["grad"], state["lobes"]


# ---------------------------------------------------------------- what a pass cannot do without
RAY_FLOPS = 60  # one watertight triangle test
SHADE_FLOPS = 400  # a vertex: shading frame, light sample, BSDF evaluation and sampling


def _tree_flops(triangles):
    """A ray's way down a binary tree over the triangles: two box slabs a level, then the triangle it hits."""
    return 12.0 * max(1.0, math.log2(max(2, triangles))) + RAY_FLOPS


def work(case):
    kind = case["kind"]
    if kind == "cast":
        n = case["rays"]
        triangles = 2 * case["grid"] ** 2 + case["spheres"] * (5120 if case["grid"] >= 256 else 320)
        # the rays, the results, and the triangles (36 B each) that this many rays can have to look at
        out = 20 if case["ray"] == "closest" else 1
        return dict(bytes=n * (32 + out) + 36 * min(triangles, n), flops=n * _tree_flops(triangles))
    if kind in ("render", "guided"):
        paths = case["width"] * case["height"] * (case["spp"] if kind == "guided" else case["side"] ** 2)
        triangles = {"large": 4096162, "room": 479826, "medium": 204964}.get(case.get("scene", "room"), 38)
        vertices = min(3, case["depth"]) + 1  # of a path that Russian roulette ends from its third bounce on
        flops = paths * vertices * (3 * _tree_flops(triangles) + SHADE_FLOPS)
        if kind == "guided":
            flops += paths * 2 * 40960
        return dict(bytes=12 * case["width"] * case["height"] + 36 * min(triangles, paths), flops=flops)
    if kind == "batch":
        paths = [int(f.config["render_region"][2]) * int(f.config["render_region"][3]) *
                 int(f.config["x_pixel_sample_count"]) ** 2 for f in _batch(case["first"], case["scenes"])]
        triangles = [f.triangle_count for f in _batch(case["first"], case["scenes"])]
        pixels = sum(int(f.config["render_region"][2]) * int(f.config["render_region"][3])
                     for f in _batch(case["first"], case["scenes"]))
        return dict(bytes=12 * pixels + 36 * sum(triangles),
                    flops=sum(p * 4 * (3 * _tree_flops(t) + SHADE_FLOPS) for p, t in zip(paths, triangles)))
    infer, train = case["infer_rows"], case["train_rows"]
    return dict(bytes=infer * (48 + 160) + train * 64 + 2 * 4 * native.GUIDE_PARAMS,
                flops=infer * 40960.0 + train * 106496.0)


# ---------------------------------------------------------------- in 64 bits
def _exact_cast(case, seed):
    """Every ray against every triangle: the hit parameter and barycentrics of the nearest one."""
    s = _cast_scene(case["grid"], case["spheres"])
    rays = _rays(s, case["rays"], case["ray"], seed).double()
    tri = []
    for o in s.objects:
        m = s.meshes[int(o["mesh_index"])]
        to_world = np.asarray(o["object_to_world"], np.float64).reshape(3, 4)
        v = m.vertices.astype(np.float64) @ to_world[:, :3].T + to_world[:, 3]
        tri.append(v[m.indices])
    tri = torch.from_numpy(np.concatenate(tri)).cuda()
    a, e1, e2 = tri[:, 0], tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0]
    t_out, bary = [], []
    for part in rays.split(max(1, (1 << 23) // tri.shape[0])):
        o, tmax, d = part[:, None, 0:3], part[:, 3], part[:, None, 4:7]
        p = torch.linalg.cross(d.expand(-1, tri.shape[0], -1), e2[None].expand(part.shape[0], -1, -1))
        det = (p * e1).sum(-1)
        q = o - a
        u = (q * p).sum(-1) / det
        r = torch.linalg.cross(q, e1[None].expand(part.shape[0], -1, -1))
        v = (d * r).sum(-1) / det
        t = (e2 * r).sum(-1) / det
        hit = (det != 0) & (u >= 0) & (v >= 0) & (u + v <= 1) & (t > 0) & (t < tmax[:, None])
        t = torch.where(hit, t, tmax[:, None])
        best, k = t.min(1)
        some = hit.gather(1, k[:, None])[:, 0]
        t_out.append(best)
        bary.append(torch.stack([u.gather(1, k[:, None])[:, 0], v.gather(1, k[:, None])[:, 0]], 1) * some[:, None])
    return torch.cat(t_out), None, None, torch.cat(bary)


def _exact_network(case, seed):
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    params = torch.from_numpy(_network_params(seed)).cuda().double().requires_grad_()
    w = [params[0:8192].view(64, 128)] + [params[8192 + 4096 * k:12288 + 4096 * k].view(64, 64) for k in range(3)]
    queries, samples = _rows(case["infer_rows"], 12, g).double(), _rows(case["train_rows"], 16, g).double()
    lo, hi = torch.tensor(BOX[:3], device="cuda").double(), torch.tensor(BOX[3:], device="cuda").double()

    def mixture(rows):
        p = (rows[:, 0:3] - lo) / (hi - lo)
        cols = []
        for k in range(16):
            f = float(np.float32(2.0 ** ((k % 3) / 3.0))) * 2.0 ** (k // 3)
            for c in range(3):
                cols += [torch.sin(math.pi * f * p[:, c]), torch.cos(math.pi * f * p[:, c])]
        h = torch.zeros((rows.shape[0], 128), dtype=torch.float64, device="cuda")
        h[:, 0:96] = torch.stack(cols, 1)
        h[:, 96:102] = rows[:, 3:9]
        h[:, 127] = 1.0
        for k in range(3):
            a = torch.relu(h @ w[k].t())
            h = torch.cat([a[:, :63], torch.ones_like(a[:, 63:])], 1)
        o = (h @ w[3].t())[:, :40].reshape(-1, 8, 5)
        mu = o[:, :, 0:3] / (o[:, :, 0:3].norm(dim=2, keepdim=True) + 1e-6)
        return mu, torch.exp(o[:, :, 3].clamp(-3.0, 8.0)), torch.log_softmax(o[:, :, 4], 1)

    loss = 0.0
    for part in samples.split(1 << 16):
        mu, kappa, log_pi = mixture(part)
        c = (mu * part[:, None, 9:12]).sum(2)
        log_c = torch.log(kappa) - math.log(2 * math.pi) - torch.log1p(-torch.exp(-2 * kappa))
        log_q = torch.logsumexp(log_pi + log_c + kappa * (c - 1), 1)
        piece = -(part[:, 12] / case["train_rows"] * log_q).sum()
        piece.backward()
        loss += float(piece.detach())
    lobes = []
    with torch.no_grad():
        for part in queries.split(1 << 16):
            mu, kappa, log_pi = mixture(part)
            lobes.append(torch.cat([mu, kappa[:, :, None], log_pi.exp()[:, :, None]], 2).reshape(-1, 40))
    return loss, params.grad, torch.cat(lobes)


def exact(case, seed):
    if case["kind"] == "network":
        return _exact_network(case, seed)
    if case["kind"] == "cast" and case["ray"] == "closest":
        triangles = 2 * case["grid"] ** 2 + case["spheres"] * 5120
        if triangles * case["rays"] <= 1 << 30:
            return _exact_cast(case, seed)
    return None  # a Monte Carlo image, or a batch too large to test every triangle
