"""Batches traced by groups of eight lanes (at most 65,536 rays) give the bytes of the kernel with one
thread per ray (which RAY_COUNT_STATS and larger batches take): leaf sizes, deep trees, batch sizes
around a block and around the limit, culling, degenerate and bounded rays; and path-traced images do not
depend on which of the two traced a wave."""
import numpy as np
import pytest
import torch

from vierkant_gb300 import geometry
from vierkant_gb300._lib import RAY_COUNT_STATS, RAY_CULL_BACK_FACES
from vierkant_gb300.pathtracer import PBRPathTracer, Scene, cornell_lights
from vierkant_gb300.raytracing import BVH

pytestmark = pytest.mark.gpu

LIMIT = 1 << 16


def _rays(n, seed, extent=1.2):
    r = np.random.default_rng(seed)
    rays = np.empty((n, 8), np.float32)
    rays[:, 0:3] = r.uniform(-extent, extent, (n, 3))
    rays[:, 3] = r.choice([0.0, 1e-4, 0.3, -0.5, -0.0], n)
    rays[:, 4:7] = r.normal(size=(n, 3))
    rays[:, 7] = r.choice([1e4, np.inf, 0.7, 0.2], n)
    rays[::7, 4] = 0.0
    rays[::11, 5] = -0.0
    rays[3::97, 4:7] = (0.0, 0.0, -1.0)
    rays[5::101, 4:7] = 0.0
    rays[6::103, 7] = -1.0
    rays[7::107, 0] = np.nan
    return torch.from_numpy(rays).cuda()


def _meshes():
    sc = geometry.cornell_scene(7, 2, 12, 8)
    yield "cornell", sc["xyz"], sc["indices"]
    yield "icosphere", *geometry.icosphere(1.0, 3)
    # triangles shrinking by 0.8 toward a corner, many of them: a tree deeper than ten levels
    r = np.random.default_rng(3)
    s = 0.8 ** r.uniform(0, 60, 30000)
    xyz = (s[:, None, None] * (1.0 + 0.1 * r.normal(size=(30000, 3, 3)))).astype(np.float32).reshape(-1, 3)
    yield "deep", xyz, np.arange(90000, dtype=np.uint32).reshape(-1, 3)


@pytest.mark.parametrize("leaf_max", [1, 2, 5, 16])
def test_group_queries_equal_thread_queries(ctx, leaf_max):
    for name, xyz, idx in _meshes():
        b = BVH(ctx, torch.from_numpy(np.ascontiguousarray(xyz)).cuda(),
                torch.from_numpy(np.ascontiguousarray(idx).astype(np.int32)).cuda(), leaf_max=leaf_max)
        if name == "deep":
            assert b.info().depth > 10 or leaf_max > 2
        for n in (1, 15, 16, 17, 4099, LIMIT, LIMIT + 1):
            rays = _rays(n, n + leaf_max)
            for flags in (0, RAY_CULL_BACK_FACES):
                for query in (b.closest_hit, b.any_hit):
                    got, want = query(rays, flags=flags), query(rays, flags=flags | RAY_COUNT_STATS)
                    assert torch.equal(got, want), (name, n, flags, query)
        b.close()
    ctx.stats(reset=True)


@pytest.mark.parametrize("lit", [False, True])
def test_images_do_not_depend_on_the_wave(ctx, lit):
    sc = geometry.cornell_scene(11, 2, 16, 8)
    mats = geometry.showcase_materials(sc["materials"]) if lit else sc["materials"]
    scene = Scene(ctx, sc["xyz"], sc["indices"], sc["tri_material"], mats, torch.full((16, 32, 3), 0.7, device="cuda"))
    if lit:
        scene.set_lights(cornell_lights())
    cam = geometry.camera_lookat((0, 0, 3.4), (0, 0, 0), (0, 1, 0), 45.0, 129, 67)
    images = []
    # waves of 8,643 and 259,290 paths (groups alone) and of 553,152 (a thread per ray, groups for what
    # the later bounces leave)
    for per_wave in (1, 30, 64):
        s = PBRPathTracer.default_settings()
        s.num_samples, s.max_trace_depth, s.rr_start_depth, s.samples_per_wave = 64, 6, 2, per_wave
        s.resolution[0], s.resolution[1] = 129, 67
        pt = PBRPathTracer(ctx, seed=5, settings=s)
        images.append(pt.render_scene(scene, cam).clone())
        pt.close()
    assert torch.isfinite(images[0]).all() and float(images[0].mean()) > 0.01
    assert torch.equal(images[0], images[1]) and torch.equal(images[0], images[2])
    scene.close()


@pytest.mark.parametrize("segments", [1, 6])
def test_alpha_images_do_not_depend_on_the_wave(ctx, segments):
    """masked and blended materials: groups trace waves of 8,643 and 259,290 paths, a thread per ray one of 553,152"""
    sc = geometry.cornell_scene(11, 2, 16, 8)
    scene = Scene(ctx, sc["xyz"], sc["indices"], sc["tri_material"], geometry.alpha_materials(sc["materials"]),
                  torch.full((16, 32, 3), 0.7, device="cuda"))
    uv, tangents = geometry.cornell_texcoords(sc)
    scene.set_normals(geometry.cornell_vertex_normals(sc))
    scene.set_texcoords(uv)
    scene.set_tangents(tangents)
    scene.set_textures(geometry.alpha_textures())
    cam = geometry.camera_lookat((0, 0, 3.4), (0, 0, 0), (0, 1, 0), 45.0, 129, 67)
    images = []
    for per_wave in (1, 30, 64):
        s = PBRPathTracer.default_settings()
        s.num_samples, s.max_trace_depth, s.rr_start_depth, s.samples_per_wave = 64, segments, 2, per_wave
        s.resolution[0], s.resolution[1] = 129, 67
        pt = PBRPathTracer(ctx, seed=5, settings=s)
        images.append(pt.render_scene(scene, cam).clone())
        pt.close()
    assert torch.isfinite(images[0]).all() and float(images[0].mean()) > 0.01
    assert torch.equal(images[0], images[1]) and torch.equal(images[0], images[2])
    scene.close()
