"""The radiance cache's encoding, hash-grid gradients and weight gradients at ragged record counts (one
record, around the 64-record CTA and chunk, several chunks per CTA) and level counts."""
import ctypes as C

import numpy as np
import pytest
import torch

from nrc_reference import encode, forward, level_resolutions, random_features, relative_l2, split_weights
from vierkant_gb300.nrc import NeuralRadianceCache
from vierkant_gb300.raytracing import _cudart

pytestmark = pytest.mark.gpu

COUNTS = [1, 63, 64, 65, 129, 64 * 152 + 1, 64 * 152 * 2 + 77]


def _read(address, count):
    out = torch.empty(count, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    assert _cudart().cudaMemcpy(C.c_void_p(out.data_ptr()), C.c_void_p(address), C.c_size_t(4 * count), 3) == 0
    return out


def _cache(ctx, levels):
    cfg = NeuralRadianceCache.default_config()
    cfg.levels, cfg.log2_table_size = levels, 12
    cache = NeuralRadianceCache(ctx, cfg)
    i = cache.info()
    g = torch.Generator(device="cuda").manual_seed(levels)
    grid = torch.rand(i.num_grid_params, generator=g, device="cuda") * 2 - 1
    cache.load_params(None, grid)
    torch.cuda.synchronize()
    return cache, _read(i.d_mlp_params, i.num_mlp_params), grid


def _reference_inputs(cfg, feats, grid, levels):
    """the 80 inputs; the columns of levels past the cache's count are zero"""
    res = level_resolutions(levels) if levels > 1 else [16]
    x = encode(feats, grid, res, 1 << cfg.log2_table_size, list(cfg.scene_min), list(cfg.scene_max), half_grid=False)
    pad = torch.zeros((x.shape[0], 32 - 2 * levels), dtype=x.dtype, device=x.device)
    return torch.cat([x[:, :2 * levels], pad, x[:, 2 * levels:]], dim=1)[:, :80]


@pytest.mark.parametrize("n", COUNTS)
@pytest.mark.parametrize("levels", [16, 5])
def test_gradients(ctx, n, levels):
    """against FP64 autograd of the same network: BF16 activations (8 bits) through six layers give
    gradients of the right direction; the cosine bound is the one of the full-size gradient tests"""
    cache, mlp, grid = _cache(ctx, levels)
    feats = random_features(n, n)
    targets = torch.rand((n, 3), generator=torch.Generator(device="cuda").manual_seed(n), device="cuda")
    cache.backward(feats, targets)
    i = cache.info()
    assert i.kernel_error == 0
    w, gr = mlp.double().requires_grad_(True), grid.double().requires_grad_(True)
    y = forward(_reference_inputs(cache.config, feats, gr, levels), split_weights(w), emulate_bf16=False)
    gw, gg = torch.autograd.grad(relative_l2(y, targets.double()), (w, gr))
    for got, want in ((_read(i.d_mlp_grads, i.num_mlp_params), gw), (_read(i.d_grid_grads, i.num_grid_params), gg)):
        got = got.double()
        assert torch.isfinite(got).all()
        cos = float((got * want).sum() / (got.norm() * want.norm()))
        assert cos > 0.99
        assert abs(float(got.norm() / want.norm()) - 1) < 0.05
    cache.close()


@pytest.mark.parametrize("n", COUNTS)
def test_inference(ctx, n):
    cache, mlp, grid = _cache(ctx, 16)
    feats = random_features(n, n + 1)
    got = cache.infer(feats).double().cpu().numpy()
    x = _reference_inputs(cache.config, feats, grid.to(torch.float16).double(), 16)
    want = forward(x, split_weights(mlp.double())).cpu().numpy()
    # the emulated BF16 network: only FP32 sums and a rounding flip of a BF16 activation (2^-8 of it) differ
    assert np.abs(got - want).max() <= 0.05 * max(1.0, np.abs(want).max())
    cache.close()


def test_binned_batches_equal_their_parts(ctx):
    """a batch of 2^19 records or more is encoded in the order of its cells; its predictions are those of
    the same records in smaller batches, records outside the box and repeated ones among them"""
    cache, _, _ = _cache(ctx, 16)
    n = (1 << 19) + 1077
    feats = random_features(n, 3)
    feats[::17, 0:3] *= 3.0
    feats[5::1000] = feats[4]
    whole = cache.infer(feats)
    half = n // 2
    assert torch.equal(whole, torch.cat([cache.infer(feats[:half]), cache.infer(feats[half:])]))
    # all in one cell: the batch keeps its order
    feats[:, 0:3] = feats[:, 0:3] * 0.01 + 0.013
    whole = cache.infer(feats)
    assert torch.equal(whole, torch.cat([cache.infer(feats[:half]), cache.infer(feats[half:])]))
    cache.close()


def _write(address, values):
    torch.cuda.synchronize()
    assert _cudart().cudaMemcpy(C.c_void_p(address), C.c_void_p(values.data_ptr()), C.c_size_t(4 * values.numel()), 3) == 0


@pytest.mark.parametrize("steps", [1, 2, 5])
@pytest.mark.parametrize("levels, kernel", [(1, 1), (16, 1), (16, 2)])
def test_adam_steps(ctx, steps, levels, kernel):
    """parameters after some steps against the formula in 64 bits. Gradients keep their sign, so nothing
    cancels: each step adds 3 roundings (2^-24) to m and 4 to v (halved by the root), the update has 8
    (4 of its own, at most 4 of the shared factor), each 1 - beta^t is off by at most 4 units of 2^-24
    (powf is good to 2 ulp), and the sum rounds the parameter. A third of the gradients is always zero and
    a third zero in every other step. The packed weights and the FP16 grid are those of the parameters."""
    cfg = NeuralRadianceCache.default_config()
    cfg.levels, cfg.log2_table_size, cfg.infer_kernel = levels, 12, kernel
    cache = NeuralRadianceCache(ctx, cfg)
    i = cache.info()
    mlp, grid = _read(i.d_mlp_params, i.num_mlp_params), _read(i.d_grid_params, i.num_grid_params)
    gen = torch.Generator(device="cuda").manual_seed(steps)
    state = []
    for p in (mlp, grid):
        base = (torch.rand(p.numel(), generator=gen, device="cuda") + 0.25) * torch.where(p < 0, -1e-3, 1e-3)
        state.append({"p": p.double(), "g": base, "kind": torch.arange(p.numel(), device="cuda") // 7 % 3,
                      "m": torch.zeros_like(p, dtype=torch.float64), "v": torch.zeros_like(p, dtype=torch.float64),
                      "tol": torch.zeros_like(p, dtype=torch.float64)})
    b1, b2, lr, eps = (float(np.float32(x)) for x in (cfg.beta1, cfg.beta2, cfg.learning_rate, cfg.epsilon))
    u = 2.0 ** -24
    for t in range(1, steps + 1):
        c1, c2 = 1 - b1 ** t, 1 - b2 ** t
        for s, address in zip(state, (i.d_mlp_grads, i.d_grid_grads)):
            g = torch.where((s["kind"] == 0) | ((s["kind"] == 1) & (t % 2 == 0)), 0.0, s["g"]) * (1 + 0.1 * t)
            _write(address, g)
            g = g.double()
            s["m"] = b1 * s["m"] + (1 - b1) * g
            s["v"] = b2 * s["v"] + (1 - b2) * g * g
            d = lr * (s["m"] / c1) / (torch.sqrt(s["v"] / c2) + eps)
            s["p"] = s["p"] - d
            s["tol"] += u * (d.abs() * (4 / c1 + 2 / c2 + 3 * t + 2 * t + 8) + s["p"].abs())
        cache.adam_step()
        torch.cuda.synchronize()
    i = cache.info()
    assert i.step == steps and i.kernel_error == 0
    got = [_read(i.d_mlp_params, i.num_mlp_params), _read(i.d_grid_params, i.num_grid_params)]
    for s, p in zip(state, got):
        assert torch.all((p.double() - s["p"]).abs() <= s["tol"])
    for address, count in ((i.d_mlp_grads, i.num_mlp_params), (i.d_grid_grads, i.num_grid_params)):
        assert torch.count_nonzero(_read(address, count)) == 0
    feats = random_features(300, 1)
    other = NeuralRadianceCache(ctx, cfg)
    other.load_params(*got)
    assert torch.equal(cache.infer(feats), other.infer(feats))


@pytest.mark.parametrize("n", [127, 128, 129, 128 * 152 + 1, 128 * 304 + 1, 45_000, 70_001])
def test_training_tiles_match_mma(ctx, n):
    """the fused tcgen05 training pass, whose intermediates are stored by tiles, against the mma.sync kernels, which
    store them by records: tiles and warpgroups at their edges. Both round every activation and layer
    gradient to BF16 (2^-8) from FP32 sums of another order; the bounds are those of the full-size comparison"""
    gen = torch.Generator(device="cuda").manual_seed(n)
    feats = random_features(n, n)
    targets = torch.rand((n, 3), device="cuda", generator=gen)
    got = {}
    for kernel in (2, 3):
        cfg = NeuralRadianceCache.default_config()
        cfg.log2_table_size, cfg.train_kernel = 12, kernel
        cache = NeuralRadianceCache(ctx, cfg)
        i = cache.info()
        gen.manual_seed(5)
        cache.load_params(torch.randn(i.num_mlp_params, device="cuda", generator=gen) * 0.2,
                          torch.randn(i.num_grid_params, device="cuda", generator=gen) * 0.5)
        cache.backward(feats, targets)
        i = cache.info()
        assert i.kernel_error == 0 and i.train_kernel == kernel
        got[kernel] = _read(i.d_mlp_grads, i.num_mlp_params), _read(i.d_grid_grads, i.num_grid_params)
        cache.close()
    for a, b in zip(got[2], got[3]):
        assert float((a * b).sum() / (a.norm() * b.norm())) > 0.9999
    assert (got[2][0] - got[3][0]).abs().max().item() <= 2e-2 * got[2][0].abs().max().item()
