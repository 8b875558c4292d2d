"""The BVH build at the sizes where its kernels change their split: one block, two and many blocks of
the collapse, full and ragged rounds; every node and triangle record equals the CPU statement."""
import ctypes as C

import numpy as np
import pytest
import torch

import oracle
from vierkant_gb300.raytracing import BVH, _cudart

pytestmark = pytest.mark.gpu


def _device_bytes(address, nbytes):
    out = torch.empty(nbytes, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    assert _cudart().cudaMemcpy(C.c_void_p(out.data_ptr()), C.c_void_p(address), C.c_size_t(nbytes), 3) == 0
    return out.cpu().numpy().tobytes()


def _mesh(n, kind):
    r = np.random.default_rng(n)
    at = r.normal(size=(n, 1, 3))
    if kind == "clustered":  # most triangles in a few tight clusters: many equal Morton codes, deep levels
        at = r.normal(size=(7, 1, 3))[r.integers(0, 7, n)] + 1e-4 * r.normal(size=(n, 1, 3))
    xyz = (at + 0.02 * r.normal(size=(n, 3, 3))).astype(np.float32).reshape(-1, 3)
    return xyz, np.arange(3 * n, dtype=np.uint32).reshape(n, 3)


@pytest.mark.parametrize("n,kind,leaf_max", [(1, "spread", 2), (2, "spread", 1), (9, "spread", 2), (2048, "spread", 2),
                                             (2049, "clustered", 1), (4095, "spread", 4), (4097, "clustered", 2),
                                             (8193, "spread", 3), (70001, "clustered", 2), (400001, "spread", 2)])
def test_build_equals_the_cpu_statement(ctx, n, kind, leaf_max):
    xyz, idx = _mesh(n, kind)
    b = BVH(ctx, torch.from_numpy(xyz).cuda(), torch.from_numpy(idx.astype(np.int32)).cuda(), leaf_max=leaf_max)
    cb = oracle.CpuBVH(xyz, idx, leaf_max)
    inf = b.info()
    assert (inf.num_nodes, inf.depth) == (cb.b.num_nodes, cb.b.depth)
    assert np.frombuffer(_device_bytes(inf.d_sorted, 4 * n), np.uint32).tobytes() == cb.sorted_prim.tobytes()
    assert _device_bytes(inf.d_nodes, 96 * inf.num_nodes) == cb.node_bytes()
    assert _device_bytes(inf.d_tris, 48 * n) == cb.tri_bytes()
    b.close()


def test_destroying_a_bvh_waits_for_its_queries(ctx):
    """a BVH destroyed right after a query was queued on it: the query still reads the tree (a destroy
    that did not wait handed the memory back under it)"""
    xyz, idx = _mesh(60000, "spread")
    x, i = torch.from_numpy(xyz).cuda(), torch.from_numpy(idx.astype(np.int32)).cuda()
    g = torch.Generator(device="cuda").manual_seed(1)
    rays = torch.randn((1_000_000, 8), generator=g, device="cuda")
    rays[:, 3], rays[:, 7] = 0.0, 1e30
    keep = BVH(ctx, x, i)
    want = keep.closest_hit(rays)
    for _ in range(3):
        b = BVH(ctx, x, i)
        got = b.closest_hit(rays)
        b.close()
        assert torch.equal(got, want)
    keep.close()
