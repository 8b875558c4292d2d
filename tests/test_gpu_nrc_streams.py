"""Inference orders its records with scratch of the cache's own: a large ray query that waits on another stream
of the same context does not hold it up."""
import pytest
import torch

from nrc_reference import random_features
from vierkant_gb300 import geometry
from vierkant_gb300.nrc import NeuralRadianceCache
from vierkant_gb300.raytracing import BVH

pytestmark = pytest.mark.gpu


def test_inference_does_not_wait_for_a_ray_query(ctx):
    n = (1 << 19) + 77
    xyz, idx = geometry.icosphere(1.0, 3)
    bvh = BVH(ctx, torch.from_numpy(xyz).cuda(), torch.from_numpy(idx.astype("int32")).cuda())
    g = torch.Generator(device="cuda").manual_seed(3)
    rays = torch.rand((n, 8), device="cuda", generator=g) * 4 - 2
    rays[:, 3], rays[:, 7] = 0.0, 1e4
    cache = NeuralRadianceCache(ctx, NeuralRadianceCache.default_config())
    feats = random_features(n, seed=5)
    want_hits, want = bvh.closest_hit(rays).clone(), cache.infer(feats).clone()
    hits, a, b = torch.empty_like(want_hits), torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(a):
        torch.cuda._sleep(1_000_000_000)  # about half a second
        bvh.closest_hit(rays, hits)
    with torch.cuda.stream(b):
        got = cache.infer(feats)
    b.synchronize()
    assert not a.query()  # the ray query is still to come
    a.synchronize()
    assert torch.equal(hits, want_hits) and torch.equal(got, want)
    cache.close()
    bvh.close()
