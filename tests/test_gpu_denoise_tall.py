"""Images of more rows than one grid of the denoiser is high (65,535 blocks of 4 x 2 rows), up to the 1,048,560 rows
that post-FX takes, against the C restatement."""
import numpy as np
import pytest
import torch

import oracle
from vierkant_gb300.pathtracer import PIXEL_DTYPE, denoise

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(1, 524_281), (1, 1_048_560)])
def test_tall_images(ctx, size):
    w, h = size
    r = np.random.default_rng(h)
    rec = np.zeros((h, w), PIXEL_DTYPE)
    rec["radiance"] = r.exponential(0.5, (h, w, 3))
    rec["depth"] = r.choice([0.0, 0.2, 0.21, 0.7], (h, w))
    rec["normal"] = r.choice(r.integers(0, 2 ** 32, 5, dtype=np.uint32), (h, w))
    rec["albedo"] = r.integers(64, 256, (h, w, 4), dtype=np.uint8).view(np.uint32)[..., 0]
    px = torch.from_numpy(rec.view(np.uint8).reshape(h, w, 32).copy()).cuda()
    got, want = denoise(ctx, px, w, h).cpu().numpy(), oracle.denoise(rec)
    # the bound of the full-frame comparison: FP32 sums of 25 taps over five passes
    assert (np.abs(got - want) / np.maximum(np.abs(want), 1e-3)).max() < 2e-4
