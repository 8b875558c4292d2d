"""World boxes of instances (the union of the mesh's boxes two levels below its root, transformed in 64 bits and
rounded outward) over transforms of every kind: one instance at a time, its box is the two-level BVH's scene box."""
import ctypes as C

import numpy as np
import pytest
import torch

from vierkant_gb300 import geometry
from vierkant_gb300.raytracing import BVH, INSTANCE_DTYPE, TLAS, _cudart

pytestmark = pytest.mark.gpu


def _nodes(bvh):
    i = bvh.info()
    out = np.empty((i.num_nodes, 24), np.uint32)
    torch.cuda.synchronize()
    assert _cudart().cudaMemcpy(C.c_void_p(out.ctypes.data), C.c_void_p(i.d_nodes), C.c_size_t(out.nbytes), 2) == 0
    return out


def _child_box(w, k):
    origin = w[:3].view(np.float32).astype(np.float64)
    scale = np.array([((int(w[3]) >> (8 * a)) & 0xFF) << 23 for a in range(3)], np.uint32).view(np.float32).astype(np.float64)
    q = w[4:16].view(np.uint8).reshape(6, 8)[:, k].astype(np.float64)
    return origin + q[:3] * scale, origin + q[3:] * scale


def _boxes(nodes):
    out, root = [], nodes[0]
    for k in range(int(root[3]) >> 24):
        c = int(root[16 + k])
        if c & 0x80000000:
            out.append(_child_box(root, k))
        else:
            out.extend(_child_box(nodes[c], g) for g in range(int(nodes[c][3]) >> 24))
    return np.array(out)


def _transforms(rng):
    eye = np.eye(3)
    turn = np.array([[0, -1, 0], [1, 0, 0], [0, 0, 1.0]])
    parts = [eye, -eye, turn, np.diag([1.0, -2.0, 0.5]), eye * 1e-3, eye * 1e6, eye + np.triu(np.ones((3, 3)), 1) * 3,
             turn @ (eye + np.tril(np.ones((3, 3)), -1))] + [rng.normal(size=(3, 3)) for _ in range(40)]
    for i, m in enumerate(parts):
        t = rng.uniform(-1, 1, 3) * [0.0, 1.0, 1e6, 1e-6][i % 4]
        yield np.concatenate([m, t[:, None]], axis=1).astype(np.float32)


@pytest.mark.parametrize("mesh", ["one", "quad", "plane", "ico"])
def test_instance_boxes(ctx, mesh):
    """each side is the 64-bit value, whose four terms may be summed in another way (2^-51 of their magnitudes),
    rounded to a neighbouring float"""
    rng = np.random.default_rng(len(mesh))
    if mesh == "ico":
        xyz, idx = geometry.icosphere(1.0, 4)[:2]
    else:
        side = {"one": 1, "quad": 1, "plane": 40}[mesh]
        u, v = np.meshgrid(np.arange(side + 1), np.arange(side + 1))
        xyz = np.stack([u.ravel(), 0 * u.ravel(), v.ravel()], axis=1).astype(np.float32)
        a = (np.arange(side)[:, None] * (side + 1) + np.arange(side)).reshape(-1, 1)
        idx = np.concatenate([a + [0, 1, side + 1], a + [1, side + 2, side + 1]])[:1 if mesh == "one" else None]
    blas = BVH(ctx, torch.from_numpy(np.ascontiguousarray(xyz, np.float32)), torch.from_numpy(np.ascontiguousarray(idx, np.int32)))
    boxes = _boxes(_nodes(blas))
    corners = np.array([[b[(m >> a) & 1][a] for a in range(3)] for b in boxes for m in range(8)])
    for T in _transforms(rng):
        inst = np.zeros(1, INSTANCE_DTYPE)
        inst[0]["transform"] = T.reshape(12)
        i = TLAS(ctx, [blas], inst).info()
        world = corners @ T[:, :3].T.astype(np.float64) + T[:, 3].astype(np.float64)
        slack = 2.0 ** -51 * (np.abs(corners) @ np.abs(T[:, :3].T.astype(np.float64)) + np.abs(T[:, 3])).max(axis=0)
        for got, want in ((np.array(i.scene_min), world.min(axis=0)), (np.array(i.scene_max), world.max(axis=0))):
            lo = np.nextafter((want - slack).astype(np.float32), np.float32(-np.inf))
            hi = np.nextafter((want + slack).astype(np.float32), np.float32(np.inf))
            assert np.all((got.astype(np.float32) >= lo) & (got.astype(np.float32) <= hi)), (mesh, T, got, want)
