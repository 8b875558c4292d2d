"""Two-level batches traced by groups of eight lanes (at most 131,072 rays) give the bytes of the kernel with
one thread per ray, which the same rays in one larger batch take: instances per leaf, coincident instances
(ties), an empty mesh, deep meshes, culling, degenerate and bounded rays; and images of an instanced scene
do not depend on the wave."""
import numpy as np
import pytest
import torch

from vierkant_gb300 import geometry
from vierkant_gb300._lib import RAY_CULL_BACK_FACES
from vierkant_gb300.pathtracer import InstancedScene, PBRPathTracer
from vierkant_gb300.raytracing import BVH, INSTANCE_DTYPE, TLAS

pytestmark = pytest.mark.gpu

LIMIT = 1 << 17


def _bvh(ctx, xyz, idx, leaf_max=2):
    return BVH(ctx, torch.from_numpy(np.ascontiguousarray(xyz)).cuda(),
               torch.from_numpy(np.ascontiguousarray(idx).astype(np.int32)).cuda(), leaf_max=leaf_max)


def _rays(n, seed):
    r = np.random.default_rng(seed)
    rays = np.empty((n, 8), np.float32)
    rays[:, 0:3] = r.uniform(-12, 12, (n, 3))
    rays[:, 3] = r.choice([0.0, 1e-3, 2.0, -1.0], n)
    rays[:, 4:7] = r.normal(size=(n, 3))
    rays[:, 7] = r.choice([1e4, np.inf, 3.0], n)
    rays[::13, 5] = 0.0
    rays[3::97, 4:7] = (0.0, 1.0, 0.0)
    rays[5::101, 4:7] = 0.0
    return torch.from_numpy(rays).cuda()


@pytest.mark.parametrize("instances,leaf_max", [(1, 4), (7, 1), (60, 16), (900, 4), (6000, 2)])
def test_group_queries_equal_thread_queries(ctx, instances, leaf_max):
    r = np.random.default_rng(1)
    s = 0.8 ** r.uniform(0, 60, 20000)
    deep = (s[:, None, None] * (1.0 + 0.1 * r.normal(size=(20000, 3, 3)))).astype(np.float32).reshape(-1, 3)
    meshes = [_bvh(ctx, *geometry.cubesphere(9, 1.0)), _bvh(ctx, *geometry.icosphere(0.7, 2), leaf_max=4),
              _bvh(ctx, np.zeros((3, 3), np.float32), np.zeros((0, 3), np.uint32)),
              _bvh(ctx, deep, np.arange(60000, dtype=np.uint32).reshape(-1, 3))]
    inst = geometry.random_instances(instances, len(meshes), (-10, -10, -10), (10, 10, 10), seed=instances, stream=5)
    inst[1::9] = inst[::9][:len(inst[1::9])]  # coincident instances: the smaller index wins
    assert inst.dtype == INSTANCE_DTYPE
    t = TLAS(ctx, meshes, inst, leaf_max=leaf_max)
    n = 2 * LIMIT + 77
    rays = _rays(n, instances)
    for flags in (0, RAY_CULL_BACK_FACES):
        for query in (t.closest_hit, t.any_hit):
            want = query(rays, flags=flags)
            for lo, hi in ((0, LIMIT), (LIMIT, 2 * LIMIT), (2 * LIMIT, n), (5, 6), (100, 117)):
                assert torch.equal(query(rays[lo:hi].contiguous(), flags=flags), want[lo:hi]), (lo, hi, flags, query)
    t.close()
    for b in meshes:
        b.close()


def test_instanced_images_do_not_depend_on_the_wave(ctx):
    st = geometry.stress_scene(terrain_n=65, num_instances=300, num_meshes=3, num_materials=16)
    scene = InstancedScene(ctx, st["meshes"], st["instances"], st["materials"], torch.full((16, 32, 3), 0.7, device="cuda"))
    cam = geometry.camera_lookat((0, 120, 300), (0, 0, 0), (0, 1, 0), 40.0, 129, 67)
    images = []
    for per_wave in (1, 30, 64):  # 8,643 / 259,290 paths (groups alone), 553,152 (both kernels)
        s = PBRPathTracer.default_settings()
        s.num_samples, s.max_trace_depth, s.rr_start_depth, s.samples_per_wave = 64, 5, 2, per_wave
        s.resolution[0], s.resolution[1] = 129, 67
        pt = PBRPathTracer(ctx, seed=5, settings=s)
        images.append(pt.render_scene(scene, cam).clone())
        pt.close()
    assert torch.isfinite(images[0]).all() and float(images[0].mean()) > 0.01
    assert torch.equal(images[0], images[1]) and torch.equal(images[0], images[2])
    scene.close()
