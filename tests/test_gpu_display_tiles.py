"""The denoiser and the bloom at image sizes around their tiles (columns of two rows per step, 32 x 28 bloom
tiles) and at every number of blur iterations per launch, against the C restatements."""
import numpy as np
import pytest
import torch

import oracle
from vierkant_gb300.pathtracer import PIXEL_DTYPE, denoise, post_fx, post_fx_settings

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("size", [(1, 5), (33, 63), (31, 64), (64, 65), (129, 131), (7, 200)])
def test_denoise_sizes(ctx, size):
    w, h = size
    r = np.random.default_rng(w * 1000 + h)
    rec = np.zeros((h, w), PIXEL_DTYPE)
    rec["radiance"] = r.exponential(0.5, (h, w, 3))
    rec["depth"] = r.choice([0.0, 0.2, 0.21, 0.7], (h, w))
    rec["normal"] = r.choice(r.integers(0, 2 ** 32, 5, dtype=np.uint32), (h, w))
    # (albedo from 0.25 up: the demodulated colours, whose differences the weights square, stay below 20)
    rec["albedo"] = r.integers(64, 256, (h, w, 4), dtype=np.uint8).view(np.uint32)[..., 0]
    px = torch.from_numpy(rec.view(np.uint8).reshape(h, w, 32).copy()).cuda()
    out, depth = denoise(ctx, px, w, h, with_depth=True)
    assert np.array_equal(depth.cpu().numpy(), rec["depth"])
    got, want = out.cpu().numpy(), oracle.denoise(rec)
    # the bound of the full-frame comparison: FP32 sums of 25 taps over five passes
    assert (np.abs(got - want) / np.maximum(np.abs(want), 1e-3)).max() < 2e-4


@pytest.mark.parametrize("iterations", [0, 1, 2, 3, 4, 7])
@pytest.mark.parametrize("size", [(1, 1), (64, 56), (66, 58), (63, 119), (131, 117)])
def test_bloom_tiles(ctx, size, iterations):
    """The threshold and each of the two passes of an iteration round the bloom b to half precision: at a
    rounding boundary either neighbour, 2^-10 b apart, may come out. Through 1 - exp(-2 (c + b)), whose
    slope times b is at most 2 x exp(-2 x) <= 0.37 (x = c + b), P roundings move the output by at most
    0.37 P 2^-10; the power 1 / 2.2 flattens it further where it matters (x -> 0: x^0.455)."""
    w, h = size
    hdr = np.random.default_rng(w * 1000 + h + iterations).exponential(0.6, (h, w, 4)).astype(np.float32)
    gamma = 1.0 if iterations % 2 else 2.2
    s = post_fx_settings(blur_iterations=iterations, gamma=gamma)
    got = post_fx(ctx, torch.from_numpy(hdr).cuda(), s).cpu().numpy()
    want = oracle.post_fx(hdr, iterations=iterations, gamma=gamma)
    assert np.abs(got - want).max() <= 0.37 * (1 + 2 * iterations) * 2.0 ** -10
    assert np.array_equal(got[..., 3], hdr[..., 3])


def test_bloom_of_a_constant_image_is_constant(ctx):
    """border and tile handling: every tap reads the same value, so every pixel is the same sum"""
    hdr = torch.full((117, 131, 4), 1.7, device="cuda")
    out = post_fx(ctx, hdr, post_fx_settings(blur_iterations=5))
    assert torch.equal(out, out[:1, :1].expand_as(out))
