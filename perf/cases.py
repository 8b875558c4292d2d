"""The work that a user of this framework has it do, as cases to time: ray queries over a BVH (device
and host buffers), acceleration-structure builds, path-traced images, the display chain and the
radiance cache.

listed() names the cases, draw(rng) gives another one of the same ranges, prepare(case, seed) makes
what a program holds before the call, run(state) is one pass through the public entry points,
work(case) the bytes and operations one pass cannot do without, exact(case, seed) its outputs in 64
bits where they are computed numbers.
"""
import math

import numpy as np
import torch

from vierkant_gb300 import geometry
from vierkant_gb300._lib import RAY_CULL_BACK_FACES
from vierkant_gb300.nrc import NeuralRadianceCache
from vierkant_gb300.pathtracer import (InstancedScene, PBRPathTracer, Scene, cornell_lights, denoise, post_fx,
                                       procedural_sky)
from vierkant_gb300.raytracing import BVH, TLAS, Context

DEV = "cuda:0"
_ctx = None


def context():
    """the one context a program keeps for its device"""
    global _ctx
    if _ctx is None:
        _ctx = Context(0)
    return _ctx


# ---- the cases ---------------------------------------------------------------------------------------

def listed():
    return [
        # mouse picking and sensor queries: a handful of rays against one object, latency only
        {"name": "pick", "kind": "trace", "query": "closest", "mesh": "ico", "detail": 5, "width": 65, "height": 63,
         "spp": 1, "bounce": False, "cull": False},
        # the ray workload of one frame: camera rays of a 720p view plus bounce rays from their hits
        {"name": "trace-frame", "kind": "trace", "query": "closest", "mesh": "cornell", "detail": 64, "width": 1280,
         "height": 720, "spp": 4, "bounce": True, "cull": False},
        # visibility of incoherent short rays (ambient occlusion baking), an odd count
        {"name": "occlusion", "kind": "trace", "query": "any", "mesh": "cornell", "detail": 64, "width": 1023,
         "height": 767, "spp": 2, "bounce": True, "cull": False},
        # a program that keeps its rays and hits in (pinned) host memory
        {"name": "trace-host", "kind": "trace", "query": "host", "mesh": "cornell", "detail": 64, "width": 1280,
         "height": 720, "spp": 2, "bounce": True, "cull": False},
        # loading or regenerating a mesh: its BVH, and the first rays against it
        {"name": "build-mesh", "kind": "build", "side": 512, "leaf_max": 2, "rays": 65536},
        # one frame of a dynamic scene: the top level rebuilt over moved instances, then the view's rays
        {"name": "dynamic-frame", "kind": "tlas", "instances": 20000, "meshes": 6, "width": 960, "height": 540},
        # an interactive preview: one sample per pixel after every camera move
        {"name": "preview", "kind": "render", "scene": "plain", "spheres": 64, "width": 321, "height": 181, "spp": 1,
         "segments": 6},
        # a still of the metal-rough scene under the sky
        {"name": "still", "kind": "render", "scene": "plain", "spheres": 64, "width": 1280, "height": 720, "spp": 16,
         "segments": 6},
        # the full material set with analytic lights
        {"name": "still-materials", "kind": "render", "scene": "showcase", "spheres": 64, "width": 853,
         "height": 480, "spp": 8, "segments": 8},
        # what a viewer does with every traced frame: denoise, bloom and tonemap
        {"name": "display", "kind": "display", "width": 1280, "height": 720},
        # the radiance cache asked for a 1080p frame's terminated paths
        {"name": "cache-infer", "kind": "infer", "queries": 2073600},
        # one optimiser step of the radiance cache on a frame's training records
        {"name": "cache-train", "kind": "train", "records": 65536, "step": True},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["trace", "trace", "build", "tlas", "render", "render", "display", "infer", "train"])
    if kind == "trace":
        query = rng.choice(["closest", "closest", "any", "host"])
        mesh = rng.choice(["ico", "cornell"])
        rays = _log_int(rng, 2000, 2_000_000)
        width = max(16, int(math.sqrt(rays * rng.uniform(0.8, 2.0))))
        return {"kind": "trace", "query": query, "mesh": mesh,
                "detail": rng.randint(2, 6) if mesh == "ico" else _log_int(rng, 2, 160), "width": width,
                "height": max(16, rays // width), "spp": rng.choice([1, 2]), "bounce": rng.random() < 0.6,
                "cull": rng.random() < 0.3}
    if kind == "build":
        return {"kind": "build", "side": _log_int(rng, 24, 720), "leaf_max": rng.choice([1, 2, 2, 4]),
                "rays": _log_int(rng, 1000, 200000)}
    if kind == "tlas":
        return {"kind": "tlas", "instances": _log_int(rng, 50, 40000), "meshes": rng.randint(1, 8),
                "width": rng.randint(100, 1100), "height": rng.randint(100, 640)}
    if kind == "render":
        scene = rng.choice(["plain", "plain", "showcase", "textured", "alpha", "media", "instanced"])
        paths = _log_int(rng, 20000, 8_000_000 if scene == "plain" else 2_000_000)
        spp = rng.choice([1, 1, 2, 4, 7])
        width = max(32, int(math.sqrt(paths / spp * rng.uniform(1.0, 2.0))))
        return {"kind": "render", "scene": scene, "spheres": _log_int(rng, 4, 100), "width": width,
                "height": max(32, paths // spp // width), "spp": spp, "segments": rng.randint(2, 8)}
    if kind == "display":
        return {"kind": "display", "width": _log_int(rng, 64, 1920), "height": _log_int(rng, 64, 1080)}
    if kind == "infer":
        return {"kind": "infer", "queries": _log_int(rng, 500, 2_000_000)}
    return {"kind": "train", "records": _log_int(rng, 300, 70000), "step": rng.random() < 0.5}


# ---- scenes and rays ---------------------------------------------------------------------------------

def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) & 0x7FFFFFFF)


def _unit(v):
    return v / v.norm(dim=-1, keepdim=True)


def _camera(width, height, seed, eye=(0.0, 0.0, 3.4), fovy=45.0):
    r = np.random.RandomState(int(seed) & 0x7FFFFFFF)
    eye = np.asarray(eye, np.float64) + r.uniform(-0.1, 0.1, 3)
    return geometry.camera_lookat(tuple(eye), (0, 0, 0), (0, 1, 0), fovy, width, height)


def _mesh(case, seed):
    if case["mesh"] == "ico":
        xyz, idx = geometry.icosphere(1.0, case["detail"])
    else:
        sc = geometry.cornell_scene(int(seed), 2, case["detail"], 16)
        xyz, idx = sc["xyz"], sc["indices"]
    return torch.from_numpy(xyz).to(DEV), torch.from_numpy(np.ascontiguousarray(idx, np.uint32).view(np.int32)).to(DEV)


def _rays(ctx, bvh, case, seed):
    """camera rays and, with "bounce", half as many rays from their hits (evenly spaced over them, in
    their order) in uniformly random directions; an any-hit query takes the bounce rays alone, cut at
    a short random distance"""
    cam = _camera(case["width"], case["height"], seed, (0.0, 0.0, 3.0 if case["mesh"] == "ico" else 3.4),
                  60.0 if case["mesh"] == "ico" else 45.0)
    prim = ctx.camera_rays(cam, int(seed), 1, case["spp"])
    if not case["bounce"]:
        return prim
    hits = bvh.closest_hit(prim)
    at = (hits[:, 0] != -1).nonzero()[:, 0]
    count = prim.shape[0] // 2
    at = at[torch.arange(count, device=DEV) * at.shape[0] // count]
    t = hits[:, 1].view(torch.float32)
    g = _generator(seed)
    d = _unit(torch.randn((count, 3), generator=g, device=DEV))
    sec = torch.empty((count, 8), device=DEV)
    sec[:, 0:3] = (prim[:, 0:3] + prim[:, 4:7] * t[:, None])[at]
    sec[:, 3] = 1e-4
    sec[:, 4:7] = d
    if case["query"] == "any":
        sec[:, 7] = torch.rand(d.shape[0], generator=g, device=DEV) * 0.5 + 0.01
        return sec.contiguous()
    sec[:, 7] = 1e4
    return torch.cat([prim, sec]).contiguous()


def _terrain(side, seed):
    """a height field of side x side vertices over [-1, 1]^2: a sum of eight octaves of random sines"""
    g = _generator(seed)
    a = torch.linspace(-1.0, 1.0, side, device=DEV)
    x, z = a[None, :].expand(side, side), a[:, None].expand(side, side)
    y = torch.zeros((side, side), device=DEV)
    for o in range(8):
        w = torch.randn(2, generator=g, device=DEV) * 2.0 ** o
        y = y + 0.2 * 2.0 ** -o * torch.sin(w[0] * x + w[1] * z + 6.28 * torch.rand(1, generator=g, device=DEV))
    xyz = torch.stack([x, y, z], dim=-1).reshape(-1, 3).contiguous()
    i = torch.arange(side * (side - 1), device=DEV, dtype=torch.int32).view(side - 1, side)[:, :-1]
    quads = torch.stack([i, i + side, i + 1, i + 1, i + side, i + side + 1], dim=-1)
    return xyz, quads.reshape(-1, 3).contiguous()


def _down_rays(n, seed):
    g = _generator(seed + 1)
    rays = torch.empty((n, 8), device=DEV)
    o = torch.rand((n, 3), generator=g, device=DEV) * 2.0 - 1.0
    o[:, 1] = 1.5
    rays[:, 0:3] = o
    rays[:, 3] = 0.0
    d = torch.randn((n, 3), generator=g, device=DEV) * 0.5
    d[:, 1] = -1.0
    rays[:, 4:7] = _unit(d)
    rays[:, 7] = 1e30
    return rays


def _settings(case):
    s = PBRPathTracer.default_settings()
    s.num_samples, s.max_trace_depth, s.rr_start_depth = case["spp"], case["segments"], 3
    s.resolution[0], s.resolution[1] = case["width"], case["height"]
    return s


def _scene(ctx, case, seed):
    kind = case["scene"]
    if kind == "instanced":
        st = geometry.stress_scene(terrain_n=129, num_instances=20 * case["spheres"], num_meshes=4, num_materials=32,
                                   seed=int(seed))
        env = procedural_sky(ctx, 512, 256)
        return InstancedScene(ctx, st["meshes"], st["instances"], st["materials"], env), \
            _camera(case["width"], case["height"], seed, (0.0, 120.0, 300.0), 40.0)
    sc = geometry.cornell_scene(int(seed), 2, case["spheres"], 16)
    env = procedural_sky(ctx, 2048, 1024) if kind == "plain" else torch.full((64, 128, 3), 0.1, device=DEV)
    mats = {"plain": lambda m: m, "showcase": geometry.showcase_materials, "textured": geometry.textured_materials,
            "alpha": geometry.alpha_materials, "media": geometry.media_materials}[kind](sc["materials"])
    scene = Scene(ctx, sc["xyz"], sc["indices"], sc["tri_material"], mats, env)
    if kind in ("showcase", "media"):
        scene.set_lights(cornell_lights())
    if kind in ("textured", "alpha"):
        uv, tangents = geometry.cornell_texcoords(sc)
        scene.set_normals(geometry.cornell_vertex_normals(sc))
        scene.set_texcoords(uv)
        scene.set_tangents(tangents)
        scene.set_textures(geometry.test_textures() if kind == "textured" else geometry.alpha_textures())
    return scene, _camera(case["width"], case["height"], seed)


# ---- pixel records -----------------------------------------------------------------------------------

def _pixel_records(case, seed):
    """A path-traced frame's pixel records: a floor and spheres in front of a sky, normals and depth of
    the geometry, checkered albedo, noisy HDR radiance with a few fireflies. uint8 [h, w, 32]."""
    h, w, g = case["height"], case["width"], _generator(seed)
    y, x = torch.meshgrid(torch.linspace(-1, 1, h, device=DEV), torch.linspace(-1, 1, w, device=DEV), indexing="ij")
    x = x * (w / h)
    normal = torch.stack([torch.zeros_like(x), torch.ones_like(x), torch.zeros_like(x)], dim=-1)
    depth = torch.where(y > 0, 0.1 * y, torch.zeros_like(y))
    normal[y <= 0] = torch.tensor([0.0, 0.0, 1.0], device=DEV)
    obj = torch.zeros((h, w), dtype=torch.int32, device=DEV)
    c = torch.rand((12, 4), generator=g, device=DEV).cpu().numpy()
    for k in range(12):
        cx, cy, r, zz = (c[k, 0] * 2 - 1) * w / h, c[k, 1] * 2 - 1, 0.05 + 0.25 * c[k, 2], 0.1 + 0.4 * c[k, 3]
        dx, dy = (x - cx) / r, (y - cy) / r
        nz = 1 - dx * dx - dy * dy
        at = (nz > 0) & (depth < zz)
        n = torch.stack([dx, -dy, nz.clamp_min(0).sqrt()], dim=-1)
        normal[at] = n[at]
        depth = torch.where(at, zz + 0.1 * nz, depth)
        obj = torch.where(at, torch.full_like(obj, k + 1), obj)
    check = ((x * 9).floor() + (y * 9).floor()) % 2
    albedo = torch.stack([0.3 + 0.5 * check, 0.6 - 0.3 * check, 0.2 + 0.05 * obj], dim=-1).clamp(0, 1)
    light = 0.15 + 1.2 * (normal * _unit(torch.tensor([0.4, 0.7, 0.6], device=DEV))).sum(-1).clamp_min(0)
    noise = torch.exp(0.7 * torch.randn((h, w, 3), generator=g, device=DEV))
    radiance = albedo * light[..., None] * noise
    fire = torch.rand((h, w), generator=g, device=DEV) < 0.002
    radiance[fire] *= 30.0
    rec = torch.zeros((h, w, 8), dtype=torch.int32, device=DEV)
    rec[..., 0:3] = radiance.contiguous().view(torch.int32)
    rec[..., 3] = torch.ones((h, w), device=DEV).view(torch.int32)
    rec[..., 4] = depth.contiguous().view(torch.int32)
    s = 1.0 / normal.abs().sum(-1)
    px, py = normal[..., 0] * s, normal[..., 1] * s
    sx, sy = torch.where(px >= 0, 1.0, -1.0), torch.where(py >= 0, 1.0, -1.0)
    below = normal[..., 2] < 0
    px, py = torch.where(below, (1 - py.abs()) * sx, px), torch.where(below, (1 - px.abs()) * sy, py)
    qx, qy = (px * 32767).round().to(torch.int32), (py * 32767).round().to(torch.int32)
    rec[..., 5] = (qx & 0xFFFF) | (qy << 16)
    rec[..., 6] = obj
    a8 = (albedo * 255).to(torch.int32)
    rec[..., 7] = a8[..., 0] | (a8[..., 1] << 8) | (a8[..., 2] << 16) | (-1 << 24)
    return rec.contiguous().view(torch.uint8).view(h, w, 32)


# ---- radiance cache ----------------------------------------------------------------------------------

LEVELS, TABLE, BASE_RES, MAX_RES = 16, 1 << 19, 16, 2048
LAYERS = [(80, 64)] + [(64, 64)] * 4 + [(64, 16)]
# a cache late in its training: small steps
LEARNING_RATE = 4e-5


def _features(n, seed):
    """n feature records on the surfaces of a box with spheres in it: position, outgoing direction,
    normal, roughness, albedo"""
    g = _generator(seed + 2)
    p = torch.rand((n, 3), generator=g, device=DEV) * 2 - 1
    nrm = torch.zeros((n, 3), device=DEV)
    wall = torch.randint(0, 5, (n,), generator=g, device=DEV)
    for k, (axis, side) in enumerate(((0, -1.0), (0, 1.0), (1, -1.0), (1, 1.0), (2, -1.0))):
        at = wall == k
        p[:, axis] = torch.where(at, torch.full_like(p[:, axis], side), p[:, axis])
        nrm[:, axis] = torch.where(at, torch.full_like(p[:, axis], -side), nrm[:, axis])
    centre = torch.rand((64, 3), generator=g, device=DEV) * 1.4 - 0.7
    radius = torch.rand(64, generator=g, device=DEV) * 0.2 + 0.1
    k = torch.randint(0, 64, (n,), generator=g, device=DEV)
    u = _unit(torch.randn((n, 3), generator=g, device=DEV))
    ball = torch.rand(n, generator=g, device=DEV) < 0.5
    p = torch.where(ball[:, None], centre[k] + radius[k][:, None] * u, p)
    nrm = torch.where(ball[:, None], u, nrm)
    d = _unit(torch.randn((n, 3), generator=g, device=DEV))
    d = torch.where((d * nrm).sum(1, keepdim=True) < 0, -d, d)
    rest = torch.rand((n, 4), generator=g, device=DEV)
    return torch.cat([p, d, nrm, rest], dim=1).contiguous()


def _parameters(seed):
    """MLP weights ([in][out] per layer, the three used outputs of the last) and hash-grid features"""
    g = _generator(seed + 3)
    mlp = []
    for l, (k, n) in enumerate(LAYERS):
        last = l == len(LAYERS) - 1
        w = (torch.rand((k, n), generator=g, device=DEV) * 2 - 1) * math.sqrt(6.0 / (k + (3 if last else n)))
        if last:
            w[:, 3:] = 0
        mlp.append(w.reshape(-1))
    grid = torch.rand(LEVELS * TABLE * 2, generator=g, device=DEV) * 2 - 1
    return torch.cat(mlp).contiguous(), grid


def _targets(feats, seed):
    g = _generator(seed + 4)
    base = 0.5 + 0.4 * torch.sin(3.0 * feats[:, 0:3]) * feats[:, 10:13]
    return (base * torch.exp(0.5 * torch.randn(base.shape, generator=g, device=DEV))).contiguous()


class _Buffer:
    """a device buffer of the library as a tensor, which keeps its owner alive"""

    def __init__(self, owner, address, count):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (int(count),), "typestr": "<f4", "data": (int(address), False),
                                         "version": 3}


def _view(owner, address, count):
    return torch.as_tensor(_Buffer(owner, address, count), device=DEV)


# ---- prepare and run ---------------------------------------------------------------------------------

def prepare(case, seed):
    ctx, kind = context(), case["kind"]
    if kind == "trace":
        xyz, idx = _mesh(case, seed)
        bvh = BVH(ctx, xyz, idx)
        rays = _rays(ctx, bvh, case, seed)
        flags = RAY_CULL_BACK_FACES if case["cull"] else 0
        state = {"kind": case["query"], "bvh": bvh, "rays": rays, "flags": flags}
        if case["query"] == "host":
            state["rays"] = rays.cpu().pin_memory()
            state["hits"] = torch.empty((rays.shape[0], 4), dtype=torch.int32).pin_memory()
        return state
    if kind == "build":
        xyz, idx = _terrain(case["side"], seed)
        return {"kind": kind, "xyz": xyz, "idx": idx, "leaf_max": case["leaf_max"],
                "rays": _down_rays(case["rays"], seed)}
    if kind == "tlas":
        blas = []
        for k in range(case["meshes"]):
            xyz, idx = geometry.cubesphere(8 + 4 * k, 1.0)
            blas.append(BVH(ctx, torch.from_numpy(xyz).to(DEV), torch.from_numpy(idx.view(np.int32)).to(DEV)))
        inst = geometry.random_instances(case["instances"], case["meshes"], (-60, -10, -60), (60, 10, 60),
                                         seed=int(seed), stream=5)
        cam = _camera(case["width"], case["height"], seed, (0.0, 40.0, 100.0), 45.0)
        return {"kind": kind, "blas": blas, "instances": inst, "rays": ctx.camera_rays(cam, int(seed), 1, 1)}
    if kind == "render":
        scene, cam = _scene(ctx, case, seed)
        return {"kind": kind, "scene": scene, "camera": cam,
                "tracer": PBRPathTracer(ctx, seed=int(seed) & 0x7FFFFFFF, settings=_settings(case))}
    if kind == "display":
        return {"kind": kind, "pixels": _pixel_records(case, seed), "width": case["width"], "height": case["height"]}
    cfg = NeuralRadianceCache.default_config()
    cfg.learning_rate = LEARNING_RATE
    cache = NeuralRadianceCache(ctx, cfg)
    mlp, grid = _parameters(seed)
    cache.load_params(mlp, grid)
    torch.cuda.synchronize()
    if kind == "infer":
        return {"kind": kind, "cache": cache, "feats": _features(case["queries"], seed)}
    feats = _features(case["records"], seed)
    info = cache.info()
    params = {"mlp": (info.d_mlp_params, info.num_mlp_params), "grid": (info.d_grid_params, info.num_grid_params)}
    grads = {"mlp": (info.d_mlp_grads, info.num_mlp_params), "grid": (info.d_grid_grads, info.num_grid_params)}
    return {"kind": "step" if case["step"] else "backward", "cache": cache, "feats": feats,
            "targets": _targets(feats, seed),
            "out": {k: _view(cache, *v) for k, v in (params if case["step"] else grads).items()}}


def run(state):
    kind = state["kind"]
    if kind == "closest":
        return state["bvh"].closest_hit(state["rays"], flags=state["flags"])
    if kind == "any":
        return state["bvh"].any_hit(state["rays"], flags=state["flags"])
    if kind == "host":
        return state["bvh"].closest_hit_host(state["rays"], state["hits"], flags=state["flags"])
    if kind == "build":
        # the new mesh's BVH takes the old one's place (released only now: its last rays are done, as the
        # build waits for the stream)
        state["bvh"] = BVH(context(), state["xyz"], state["idx"], leaf_max=state["leaf_max"])
        return state["bvh"].closest_hit(state["rays"])
    if kind == "tlas":
        state["tlas"] = TLAS(context(), state["blas"], state["instances"])  # and the last frame's goes
        return state["tlas"].closest_hit(state["rays"])
    if kind == "render":
        state["tracer"].reset_accumulator()
        return state["tracer"].render_scene(state["scene"], state["camera"])
    if kind == "display":
        smooth = denoise(context(), state["pixels"], state["width"], state["height"])
        return {"denoised": smooth, "display": post_fx(context(), smooth)}
    if kind == "infer":
        return state["cache"].infer(state["feats"])
    if kind == "step":
        loss = state["cache"].train_step(state["feats"], state["targets"])
        return {"loss": loss, **state["out"]}
    state["cache"].backward(state["feats"], state["targets"])
    return state["out"]


# ---- what a pass cannot do without ---------------------------------------------------------------------

def _ray_flops(tris):
    """one 8-wide node per level of the tree (12 operations per child box) and one triangle test"""
    return 96.0 * max(1.0, math.log(max(tris, 2)) / math.log(8.0)) + 54.0


def work(case):
    kind = case["kind"]
    if kind == "trace":
        tris = 20 * 4 ** case["detail"] if case["mesh"] == "ico" else 10 + 3072 * case["detail"]
        prim = case["width"] * case["height"] * case["spp"]
        rays = prim if not case["bounce"] else (prim // 2 if case["query"] == "any" else prim + prim // 2)
        out = 4 if case["query"] == "any" else 16
        return {"bytes": rays * (32 + out) + 48 * tris, "flops": rays * _ray_flops(tris)}
    if kind == "build":
        tris = 2 * (case["side"] - 1) ** 2
        # vertices and indices in, triangle records and nodes (one per five triangles) out, the rays
        return {"bytes": 12 * case["side"] ** 2 + 12 * tris + 48 * tris + 96 * tris / 5 + 48 * case["rays"],
                "flops": 60 * tris + case["rays"] * _ray_flops(tris)}
    if kind == "tlas":
        n, rays = case["instances"], case["width"] * case["height"]
        return {"bytes": n * (64 + 2 * 128 + 96 / 3) + rays * (32 + 32), "flops": 300 * n + rays * _ray_flops(8 * n)}
    if kind == "render":
        pixels = case["width"] * case["height"]
        tris = 10 + 3072 * case["spheres"]
        # the image; the geometry once; at least one extension and one shadow ray per sample
        return {"bytes": 12 * pixels + 60 * tris, "flops": pixels * case["spp"] * 2 * _ray_flops(tris)}
    if kind == "display":
        pixels = case["width"] * case["height"]
        # records in, denoised image out, display image out; five passes of 25 taps and the blur
        return {"bytes": pixels * (32 + 16 + 16), "flops": pixels * (5 * 25 * 24 + 6 * 9 * 8 / 4 + 40)}
    params = sum(k * n for k, n in LAYERS)
    if kind == "infer":
        n = case["queries"]
        return {"bytes": n * (52 + 12) + min(n * 16 * 8 * 4, 2 * LEVELS * TABLE * 2), "flops": n * (2 * params + 700)}
    n = case["records"]
    touched = min(n * 16 * 8, LEVELS * TABLE)
    if case["step"]:
        # the optimiser reads and writes parameter, two moments and gradient of every grid entry
        return {"bytes": n * 64 + touched * 4 + LEVELS * TABLE * 2 * 34, "flops": n * (6 * params + 1400)}
    return {"bytes": n * 64 + touched * (4 + 16), "flops": n * (6 * params + 1400)}


# ---- outputs in 64 bits --------------------------------------------------------------------------------

def _sh(d):
    x, y, z = d[:, 0], d[:, 1], d[:, 2]
    xx, yy, zz = x * x, y * y, z * z
    c = [math.sqrt(v / math.pi) for v in (1 / 4, 3 / 4, 15 / 4, 5 / 16, 15 / 16, 35 / 32, 105 / 4, 21 / 32, 7 / 16,
                                          105 / 16)]
    return torch.stack([torch.full_like(x, c[0]), -c[1] * y, c[1] * z, -c[1] * x, c[2] * x * y, -c[2] * y * z,
                        c[3] * (3 * zz - 1), -c[2] * x * z, c[4] * (xx - yy), -c[5] * y * (3 * xx - yy),
                        c[6] * x * y * z, -c[7] * y * (5 * zz - 1), c[8] * z * (5 * zz - 3), -c[7] * x * (5 * zz - 1),
                        c[9] * z * (xx - yy), -c[5] * x * (xx - 3 * yy)], dim=1)


def _predict(feats, mlp, grid):
    """the cache's network on feature records, everything in 64 bits: a multiresolution hash grid over
    [-1, 1]^3, spherical harmonics of direction and normal, roughness, albedo; six layers with ReLU"""
    f = feats.double()
    p = ((f[:, 0:3] + 1.0) * 0.5).clamp(0, 1)
    growth = np.float32(math.exp((math.log(MAX_RES) - math.log(BASE_RES)) / (LEVELS - 1)))
    cols, res = [], np.float32(BASE_RES)
    for l in range(LEVELS):
        r = int(res)
        x = p * r
        cell = x.floor().clamp(max=r - 1)
        t, cell = x - cell, cell.to(torch.int64)
        acc = 0
        for k in range(8):
            o = [k & 1, (k >> 1) & 1, (k >> 2) & 1]
            q = [cell[:, a] + o[a] for a in range(3)]
            if (r + 1) ** 3 <= TABLE:
                at = q[0] + q[1] * (r + 1) + q[2] * (r + 1) ** 2
            else:
                at = (q[0] ^ ((q[1] * 2654435761) & 0xFFFFFFFF) ^ ((q[2] * 805459861) & 0xFFFFFFFF)) & (TABLE - 1)
            weight = 1
            for a in range(3):
                weight = weight * (t[:, a] if o[a] else 1 - t[:, a])
            acc = acc + weight[:, None] * grid.view(LEVELS, TABLE, 2)[l].index_select(0, at)
        cols.append(acc)
        res = np.float32(res * growth)
    h = torch.cat(cols + [_sh(f[:, 3:6]), _sh(f[:, 6:9]), f[:, 9:13],
                          torch.zeros((f.shape[0], 12), dtype=torch.float64, device=DEV)], dim=1)
    off = 0
    for l, (k, n) in enumerate(LAYERS):
        h = h @ mlp[off:off + k * n].view(k, n)
        off += k * n
        if l < len(LAYERS) - 1:
            h = torch.relu(h)
    return h[:, 0:3]


def _display_exact(case, seed):
    rec = _pixel_records(case, seed).view(torch.int32)
    h, w = case["height"], case["width"]
    color = rec[..., 0:3].contiguous().view(torch.float32).double()
    depth = rec[..., 4].contiguous().view(torch.float32).double()
    packed = rec[..., 5]
    qx = (((packed << 16) >> 16).double() / 32767).clamp_min(-1)
    qy = ((packed >> 16).double() / 32767).clamp_min(-1)
    nz = 1 - qx.abs() - qy.abs()
    sx, sy = torch.where(qx >= 0, 1.0, -1.0).double(), torch.where(qy >= 0, 1.0, -1.0).double()
    normal = _unit(torch.stack([torch.where(nz < 0, (1 - qy.abs()) * sx, qx),
                                torch.where(nz < 0, (1 - qx.abs()) * sy, qy), nz], dim=-1))
    a8 = rec[..., 7]
    albedo = torch.stack([((a8 >> s) & 255).double() / 255 for s in (0, 8, 16)], dim=-1).clamp_min(0.01)
    luma = torch.tensor([0.299, 0.587, 0.114], dtype=torch.float64, device=DEV)
    tap = [1 / 16, 1 / 4, 3 / 8, 1 / 4, 1 / 16]
    ys, xs = torch.arange(h, device=DEV), torch.arange(w, device=DEV)
    for step in (1, 2, 4, 8, 16):
        dm = color / albedo
        lum = dm @ luma
        total, weight = torch.zeros_like(dm), torch.zeros_like(lum)
        for j in range(5):
            for i in range(5):
                yy, xx = (ys + (j - 2) * step).clamp(0, h - 1), (xs + (i - 2) * step).clamp(0, w - 1)

                def at(v):
                    return v[yy][:, xx]
                e = (lum - at(lum)) ** 2 / 0.9 + ((normal - at(normal)) ** 2).sum(-1) / 0.3 + (depth - at(depth)).abs()
                k = torch.exp(-e) * (tap[i] * tap[j])
                total += at(dm) * k[..., None]
                weight += k
        color = total / weight[..., None] * albedo
    smooth = torch.cat([color, torch.zeros((h, w, 1), dtype=torch.float64, device=DEV)], dim=-1)

    def resize(img, oh, ow):
        ih, iw = img.shape[:2]

        def axis(n, m):
            x = (torch.arange(n, device=DEV, dtype=torch.float64) + 0.5) / n * m - 0.5
            x0 = x.floor()
            return x0.long().clamp(0, m - 1), (x0.long() + 1).clamp(0, m - 1), x - x0
        x0, x1, fx = axis(ow, iw)
        y0, y1, fy = axis(oh, ih)
        rows = img[y0] + (img[y1] - img[y0]) * fy[:, None, None]
        return rows[:, x0] + (rows[:, x1] - rows[:, x0]) * fx[None, :, None]
    bh, bw = max(h // 2, 1), max(w // 2, 1)
    b = resize(smooth, bh, bw).clamp_min(0)
    t = ((b[..., 0:3] @ luma - 0.95) / (1.1 - 0.95)).clamp(0, 1)
    s = (t * t * (3 - 2 * t))[..., None]
    b = torch.cat([b[..., 0:3] * s, 1 + (b[..., 3:4] - 1) * s], dim=-1)
    g = [math.exp(-(k - 4) ** 2 / (2 * 1.7 ** 2)) for k in range(9)]
    for _ in range(3):
        for axis, n in ((1, bw), (0, bh)):
            at = [(torch.arange(n, device=DEV) + k).clamp(0, n - 1) for k in range(-4, 5)]
            b = sum(b.index_select(axis, a) * (v / sum(g)) for a, v in zip(at, g))
    display = 1 - torch.exp(-(smooth[..., 0:3] + resize(b, h, w)[..., 0:3]) * 2.0)
    return {"denoised": smooth, "display": torch.cat([display, smooth[..., 3:4]], dim=-1)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "display":
        return _display_exact(case, seed)
    if kind not in ("infer", "train"):
        return None  # ray queries give whole numbers and bits; a traced image has no closed form
    mlp, grid = (v.double() for v in _parameters(seed))
    if kind == "infer":
        feats = _features(case["queries"], seed)
        return torch.cat([_predict(f, mlp, grid) for f in feats.split(262144)])
    feats = _features(case["records"], seed)
    target = _targets(feats, seed).double()
    mlp.requires_grad_(True)
    grid.requires_grad_(True)
    y = _predict(feats, mlp, grid)
    loss = ((y - target) ** 2 / (y.detach() ** 2 + 0.01)).mean()
    g = dict(zip(("mlp", "grid"), torch.autograd.grad(loss, (mlp, grid))))
    if not case["step"]:
        return g
    # Adam's first step: both moments are the gradient's after bias correction
    with torch.no_grad():
        new = {k: v - LEARNING_RATE * g[k] / (g[k].abs() + 1e-15) for k, v in (("mlp", mlp), ("grid", grid))}
    return {"loss": float(loss), **new}
