"""The grid barrier of the BVH build gives up after its limit in time: a build whose barriers expect a block that
does not exist returns VKG_ERR_TIMEOUT, for the fewest blocks that wait for each other and for one a SM, and the
builds after it are what they were."""
import ctypes as C
import time

import numpy as np
import pytest
import torch

import oracle
from vierkant_gb300 import _lib
from vierkant_gb300.raytracing import BVH

pytestmark = pytest.mark.gpu
LIMIT = 5_000_000  # ns
ERR_INVALID, ERR_TIMEOUT = 1, 5


@pytest.mark.parametrize("n", [2049, 400001])
def test_a_barrier_that_runs_out_ends_the_build(ctx, n):
    r = np.random.default_rng(n)
    xyz = (r.normal(size=(n, 1, 3)) + 0.02 * r.normal(size=(n, 3, 3))).astype(np.float32).reshape(-1, 3)
    idx = np.arange(3 * n, dtype=np.uint32).reshape(n, 3)
    d_xyz, d_idx = torch.from_numpy(xyz).cuda(), torch.from_numpy(idx.astype(np.int32)).cuda()
    call = _lib.lib().vkg_diag_build_timeout
    BVH(ctx, d_xyz, d_idx).close()  # first-call costs
    for _ in range(2):
        t0 = time.perf_counter()
        status = call(ctx.handle, C.c_void_p(d_xyz.data_ptr()), 3 * n, C.c_void_p(d_idx.data_ptr()), n, LIMIT,
                      C.c_void_p(ctx.stream()))
        took = time.perf_counter() - t0
        assert status == ERR_TIMEOUT and b"barrier" in _lib.lib().vkg_last_error(ctx.handle)
        assert LIMIT * 1e-9 <= took < 50 * LIMIT * 1e-9, took
    b, cb = BVH(ctx, d_xyz, d_idx, leaf_max=2), oracle.CpuBVH(xyz, idx, 2)
    assert (b.info().num_nodes, b.info().depth) == (cb.b.num_nodes, cb.b.depth)
    b.close()


def test_the_diagnostic_refuses_builds_without_a_barrier(ctx):
    xyz = torch.zeros(9, device="cuda")
    idx = torch.zeros(3, dtype=torch.int32, device="cuda")
    assert _lib.lib().vkg_diag_build_timeout(ctx.handle, C.c_void_p(xyz.data_ptr()), 3, C.c_void_p(idx.data_ptr()), 1, LIMIT,
                                             C.c_void_p(ctx.stream())) == ERR_INVALID
