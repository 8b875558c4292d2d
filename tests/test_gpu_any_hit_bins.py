"""Any-hit batches large enough to be traced in bins (3 * 2^19 rays) equal the given order, as closest-hit batches do
from 2^19 on, and images whose waves bin their shadow rays equal those of smaller waves, whose rays are
traced in the given order (a bounce's binned shadow rays share a launch with the next bounce's rays)."""
import numpy as np
import pytest
import torch

from vierkant_gb300 import geometry
from vierkant_gb300._lib import RAY_CULL_BACK_FACES, RAY_KEEP_ORDER
from vierkant_gb300.pathtracer import PBRPathTracer, Scene
from vierkant_gb300.raytracing import BVH

pytestmark = pytest.mark.gpu
BIN_MIN_ANY = 3 << 19


@pytest.mark.parametrize("n", [BIN_MIN_ANY - 1, BIN_MIN_ANY, BIN_MIN_ANY + 1, 2_000_003])
def test_any_hit_in_bins_equals_the_given_order(ctx, n):
    sc = geometry.cornell_scene(0x5EED, 2, 16, 16)
    b = BVH(ctx, torch.from_numpy(sc["xyz"]).cuda(), torch.from_numpy(sc["indices"].astype(np.int32)).cuda())
    cam = geometry.camera_lookat((0, 0, 3.4), (0, 0, 0), (0, 1, 0), 45.0, 640, 360)
    coherent = ctx.camera_rays(cam, 0x5EED, 2, 2)  # 460,800 rays, whose tiles keep their order
    g = torch.Generator(device="cuda").manual_seed(n)
    rays = torch.empty((n, 8), device="cuda")
    rays[:, 0:3] = torch.rand((n, 3), device="cuda", generator=g) * 2 - 1
    rays[:, 3] = 1e-3
    rays[:, 4:7] = torch.randn((n, 3), device="cuda", generator=g)
    rays[:, 7] = torch.rand(n, device="cuda", generator=g)  # shadow-like segments: some end before they hit
    rays[100_000:100_000 + coherent.shape[0]] = coherent
    for cull in (0, RAY_CULL_BACK_FACES):
        binned, given = b.any_hit(rays, flags=cull), b.any_hit(rays, flags=cull | RAY_KEEP_ORDER)
        assert torch.equal(binned, given)
        assert 0.05 < float(given.float().mean()) < 0.95
        # and the given order's answers, whatever kernel a batch of their size takes
        parts = torch.cat([b.any_hit(p.contiguous(), flags=cull) for p in rays.split(65_000)])
        assert torch.equal(binned, parts)
    b.close()


def test_images_with_binned_shadow_rays(ctx):
    sc = geometry.cornell_scene(11, 2, 16, 8)
    scene = Scene(ctx, sc["xyz"], sc["indices"], sc["tri_material"], sc["materials"], torch.full((16, 32, 3), 0.7, device="cuda"))
    cam = geometry.camera_lookat((0, 0, 3.4), (0, 0, 0), (0, 1, 0), 45.0, 129, 67)
    images = []
    for per_wave in (20, 100, 200):  # 172,860 / 864,300 / 1,728,600 paths; the last one's shadow rays are binned
        s = PBRPathTracer.default_settings()
        s.num_samples, s.max_trace_depth, s.rr_start_depth, s.samples_per_wave = 200, 6, 2, per_wave
        s.resolution[0], s.resolution[1] = 129, 67
        pt = PBRPathTracer(ctx, seed=5, settings=s)
        images.append(pt.render_scene(scene, cam).clone())
        pt.close()
    assert 129 * 67 * 200 > BIN_MIN_ANY
    assert torch.isfinite(images[0]).all() and float(images[0].mean()) > 0.01
    assert torch.equal(images[0], images[1]) and torch.equal(images[0], images[2])
    scene.close()
