"""Closest-hit batches over instances that overlap a lot leave the groups of eight lanes at 49,152 rays, all others at
131,072: on both sides of either line the hits are those of one large batch, which one thread per ray traces;
and the overlap that decides does not depend on the instances' scale or place."""
import numpy as np
import pytest
import torch

from vierkant_gb300 import geometry
from vierkant_gb300.raytracing import BVH, TLAS

pytestmark = pytest.mark.gpu
LINES = (3 << 14, 1 << 17)


@pytest.mark.parametrize("instances,size", [(300, 8.0), (6000, 4.0), (6000, 4000.0)])
def test_batches_around_the_lines(ctx, instances, size):
    xyz, idx = geometry.cubesphere(6, size / 8.0)
    mesh = BVH(ctx, torch.from_numpy(xyz).cuda(), torch.from_numpy(idx.view(np.int32)).cuda())
    inst = geometry.random_instances(instances, 1, (-size,) * 3, (size,) * 3, seed=7, stream=5)
    t = TLAS(ctx, [mesh], inst)
    g = torch.Generator(device="cuda").manual_seed(instances)
    n = 2 * LINES[1]
    rays = torch.empty((n, 8), device="cuda")
    rays[:, 0:3] = (torch.rand((n, 3), device="cuda", generator=g) * 2 - 1) * size
    rays[:, 3] = 1e-3 * size
    rays[:, 4:7] = torch.randn((n, 3), device="cuda", generator=g)
    rays[:, 7] = torch.rand(n, device="cuda", generator=g) * size
    for query in (t.closest_hit, t.any_hit):
        want = query(rays)
        assert 0.01 < float((want.reshape(n, -1)[:, 0] != (-1 if query == t.closest_hit else 0)).float().mean()) < 0.999
        for m in [line + k for line in LINES for k in (-1, 0, 1)]:
            assert torch.equal(query(rays[:m].contiguous()), want[:m]), (m, query)
    t.close()
    mesh.close()
