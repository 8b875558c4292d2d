"""Batches with a device-side count (a cached frame's queries): few records in a large batch are encoded in the given
order, without the work of ordering the batch, and the predictions do not depend on it."""
import ctypes as C

import pytest
import torch

from nrc_reference import random_features
from vierkant_gb300 import _lib
from vierkant_gb300.nrc import NeuralRadianceCache

pytestmark = pytest.mark.gpu
BIN_MIN = 1 << 19
CAPACITY = BIN_MIN + 77


@pytest.mark.parametrize("kernel", [1, 2])
def test_few_records_keep_their_order(ctx, kernel):
    cfg = NeuralRadianceCache.default_config()
    cfg.infer_kernel = kernel
    cache = NeuralRadianceCache(ctx, cfg)
    feats = random_features(CAPACITY, seed=6)
    want = cache.infer(feats)
    for count in (0, 1, 1000, BIN_MIN - 1, BIN_MIN, CAPACITY):
        d_n = torch.tensor([count], dtype=torch.int32, device="cuda")
        reordered = torch.full((1,), 12345, dtype=torch.int32, device="cuda")
        out = torch.full((CAPACITY, 3), float("nan"), device="cuda")
        _lib.check(_lib.lib().vkg_diag_nrc_predict(cache.handle, C.c_void_p(feats.data_ptr()), CAPACITY,
                                                   C.c_void_p(d_n.data_ptr()), C.c_void_p(out.data_ptr()),
                                                   C.c_void_p(reordered.data_ptr()), C.c_void_p(ctx.stream())), ctx.handle)
        assert (reordered.item() > 0) == (count >= BIN_MIN), count
        assert torch.equal(out[:count], want[:count]) and torch.isnan(out[count:]).all()
    cache.close()
