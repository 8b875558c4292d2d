// Bloom + tonemap composition of the path tracer's output: the reference's post-FX pass
// (src/PBRPathTracer.cpp:405-465) as headless CUDA kernels, display only.
//
//   bloom threshold   shaders/slang/fullscreen/bloom_thresh.slang: half-resolution image (Bloom's
//                     framebuffer, PBRPathTracer.cpp:797-799) of the bilinearly sampled HDR colour,
//                     max(c, 0) faded in by smoothstep(0.95, 1.1, NTSC luma) (Bloom.hpp brightness_thresh)
//   gaussian blur     src/GaussianBlur.cpp, shaders/slang/fullscreen/gaussian_blur.slang: 3 iterations
//                     (PBRPathTracer.cpp:799) of a horizontal and a vertical 9-tap Gaussian
//                     (GaussianBlur_<9>), clamp-to-edge
//   composition       shaders/slang/fullscreen/bloom_composition.slang + utils/tonemap.slang:
//                     1 - exp(-(hdr + bloom) * exposure), then pow(., 1 / gamma); alpha of the HDR image
//                     (the path tracer binds an empty motion image, so the motion blur takes one tap)
//
// The bloom images are RGBA16F as in the reference (Bloom::create_info_t::color_format), so every
// threshold / blur output is rounded to half precision. The reference's blur merges tap pairs into
// bilinear fetches; here the 9 taps are summed directly (the same convolution, without the texture
// unit's fixed-point filter weights). Texture sampling is restated as bilinear filtering with
// clamp-to-edge addressing at texel centres. The 9-tap kernel is crocore::createGaussianKernel_1D
// (crocore, a submodule absent from the reference checkout; pinned commit unknown) with sigma
// deduced from the size: restated as the normalised Gaussian exp(-x^2 / (2 sigma^2)), x = -4..4,
// sigma = 0.3 ((9 - 1) / 2 - 1) + 0.8 = 1.7.
#include "internal.hpp"

#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <type_traits>
#include <utility>

namespace vkg
{
namespace
{

// the blur's taps, normalised
struct blur_taps
{
    float w[9];
};

__device__ __forceinline__ float4 ld_half4(const __half *p)
{
    const __half2 a = reinterpret_cast<const __half2 *>(p)[0], b = reinterpret_cast<const __half2 *>(p)[1];
    const float2 fa = __half22float2(a), fb = __half22float2(b);
    return make_float4(fa.x, fa.y, fb.x, fb.y);
}
__device__ __forceinline__ void st_half4(__half *p, float4 v)
{
    reinterpret_cast<__half2 *>(p)[0] = __floats2half2_rn(v.x, v.y);
    reinterpret_cast<__half2 *>(p)[1] = __floats2half2_rn(v.z, v.w);
}

// bilinear sample at texture coordinate (u, v) in [0, 1] of a w x h image, clamp-to-edge
template<class Load>
__device__ __forceinline__ float4 bilinear(Load load, uint32_t w, uint32_t h, float u, float v)
{
    const float x = u * (float)w - 0.5f, y = v * (float)h - 0.5f;
    const float x0f = floorf(x), y0f = floorf(y);
    const float fx = x - x0f, fy = y - y0f;
    const int x0 = min(max((int)x0f, 0), (int)w - 1), x1 = min(max((int)x0f + 1, 0), (int)w - 1);
    const int y0 = min(max((int)y0f, 0), (int)h - 1), y1 = min(max((int)y0f + 1, 0), (int)h - 1);
    const float4 a = load(x0, y0), b = load(x1, y0), c = load(x0, y1), d = load(x1, y1);
    auto lerp4 = [](float4 p, float4 q, float t) {
        return make_float4(p.x + (q.x - p.x) * t, p.y + (q.y - p.y) * t, p.z + (q.z - p.z) * t, p.w + (q.w - p.w) * t);
    };
    return lerp4(lerp4(a, b, fx), lerp4(c, d, fx), fy);
}

// the thresholded HDR colour of bloom pixel (x, y)
__device__ __forceinline__ float4 bloom_threshold(const float4 *__restrict__ hdr, uint32_t w, uint32_t h, uint32_t bw,
                                                  uint32_t bh, int x, int y, float lo, float hi)
{
    const float u = ((float)x + 0.5f) / (float)bw, v = ((float)y + 0.5f) / (float)bh;
    float4 c = bilinear([&](int i, int j) { return __ldg(&hdr[(size_t)j * w + i]); }, w, h, u, v);
    c = make_float4(fmaxf(c.x, 0.f), fmaxf(c.y, 0.f), fmaxf(c.z, 0.f), fmaxf(c.w, 0.f));
    const float br = c.x * 0.299f + c.y * 0.587f + c.z * 0.114f;
    const float t = fminf(fmaxf((br - lo) / (hi - lo), 0.f), 1.f);
    const float s = t * t * (3.f - 2.f * t);
    // lerp((0, 0, 0, 1), c, s)
    return make_float4(c.x * s, c.y * s, c.z * s, 1.f + (c.w - 1.f) * s);
}

// Up to ITER blur iterations (horizontal and vertical pass each) of a 32 x 28 tile in shared memory, after
// the threshold (hdr given) or from a bloom image (in). A tile starts with a border of 4 ITER pixels
// and every pass gives up 4 of them, so that one launch replaces the threshold and two launches per
// iteration; every pass is rounded to half precision as an image would be. 640x360, three iterations: 33 us
// (seven launches) -> 22 us, bound by the latency of its seven steps (256 threads a block: 25 us).
constexpr int BLOOM_TX = 32, BLOOM_TY = 28, BLOOM_THREADS = 512; // (two tiles with borders fit 48 KB)
template<int ITER>
__global__ void __launch_bounds__(BLOOM_THREADS)
        k_bloom(const float4 *__restrict__ hdr, uint32_t w, uint32_t h, float lo, float hi,
                const __half *__restrict__ in, uint32_t bw, uint32_t bh, blur_taps taps, __half *__restrict__ out)
{
    constexpr int HALO = 4 * ITER, SX = BLOOM_TX + 2 * HALO, SY = BLOOM_TY + 2 * HALO;
    extern __shared__ __align__(16) uint2 tile[]; // two SX x SY half4 images
    const int x0 = (int)blockIdx.x * BLOOM_TX - HALO, y0 = (int)blockIdx.y * BLOOM_TY - HALO;
    __half *a = reinterpret_cast<__half *>(tile), *b = reinterpret_cast<__half *>(tile + SX * SY);
    for(int i = threadIdx.x; i < SX * SY; i += BLOOM_THREADS)
    {
        const int x = x0 + i % SX, y = y0 + i / SX;
        if(x < 0 || y < 0 || x >= (int)bw || y >= (int)bh) continue;
        if(hdr) st_half4(a + 4 * i, bloom_threshold(hdr, w, h, bw, bh, x, y, lo, hi));
        else reinterpret_cast<uint2 *>(a)[i] = __ldg(reinterpret_cast<const uint2 *>(in) + (size_t)y * bw + x);
    }
    // pixels [l, l + nx) x [t, t + ny) of the tile from `src` to `dst`
    auto pass = [&](const __half *src, __half *dst, auto vertical, int l, int t, int nx, int ny) {
        constexpr bool V = decltype(vertical)::value;
        __syncthreads();
        for(int i = threadIdx.x; i < nx * ny; i += BLOOM_THREADS)
        {
            const int px = l + i % nx, py = t + i / nx, x = x0 + px, y = y0 + py;
            if(x < 0 || y < 0 || x >= (int)bw || y >= (int)bh) continue;
            float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for(int k = -4; k <= 4; ++k)
            {
                const int q = V ? (min(max(y + k, 0), (int)bh - 1) - y0) * SX + px
                                : py * SX + min(max(x + k, 0), (int)bw - 1) - x0;
                const float4 v = ld_half4(src + 4 * q);
                const float wk = taps.w[k + 4];
                acc.x += v.x * wk;
                acc.y += v.y * wk;
                acc.z += v.z * wk;
                acc.w += v.w * wk;
            }
            st_half4(dst + 4 * (py * SX + px), acc);
        }
    };
#pragma unroll
    for(int it = 0; it < ITER; ++it)
    {
        const int m = 4 * it; // border already given up
        pass(a, b, std::false_type{}, m + 4, m, SX - 2 * m - 8, SY - 2 * m);
        pass(b, a, std::true_type{}, m + 4, m + 4, SX - 2 * m - 8, SY - 2 * m - 8);
    }
    __syncthreads();
    for(int i = threadIdx.x; i < BLOOM_TX * BLOOM_TY; i += BLOOM_THREADS)
    {
        const int px = HALO + i % BLOOM_TX, py = HALO + i / BLOOM_TX, x = x0 + px, y = y0 + py;
        if(x < (int)bw && y < (int)bh)
            reinterpret_cast<uint2 *>(out)[(size_t)y * bw + x] = reinterpret_cast<const uint2 *>(a)[py * SX + px];
    }
}

__global__ void k_composite(const float4 *__restrict__ hdr, const __half *__restrict__ bloom, uint32_t w, uint32_t h,
                            uint32_t bw, uint32_t bh, float exposure, float inv_gamma, float4 *__restrict__ out)
{
    const uint32_t x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y * blockDim.y + threadIdx.y;
    if(x >= w || y >= h) return;
    const float4 c = hdr[(size_t)y * w + x];
    float3 b = make_float3(0.f, 0.f, 0.f);
    if(bloom)
    {
        const float u = ((float)x + 0.5f) / (float)w, v = ((float)y + 0.5f) / (float)h;
        const float4 s = bilinear([&](int i, int j) { return ld_half4(bloom + 4 * ((size_t)j * bw + i)); }, bw, bh, u, v);
        b = make_float3(s.x, s.y, s.z);
    }
    float r = 1.f - expf(-(c.x + b.x) * exposure), g = 1.f - expf(-(c.y + b.y) * exposure),
          bl = 1.f - expf(-(c.z + b.z) * exposure);
    if(inv_gamma != 1.f) // (the default gamma is 1)
    {
        r = powf(r, inv_gamma);
        g = powf(g, inv_gamma);
        bl = powf(bl, inv_gamma);
    }
    out[(size_t)y * w + x] = make_float4(r, g, bl, c.w);
}

}// namespace
}// namespace vkg

using namespace vkg;

extern "C" vkg_status vkg_post_fx_default(vkg_post_fx_settings *s)
{
    if(!s) return VKG_ERR_INVALID_ARGUMENT;
    // PBRPathTracer::settings_t (PBRPathTracer.hpp:74-86), Bloom::create_info_t, PBRPathTracer.cpp:797-799
    *s = vkg_post_fx_settings{};
    s->tonemap = 1;
    s->bloom = 1;
    s->exposure = 2.f;
    s->gamma = 1.f;
    s->brightness_thresh[0] = 0.95f;
    s->brightness_thresh[1] = 1.1f;
    s->blur_iterations = 3;
    return VKG_OK;
}

extern "C" vkg_status vkg_post_fx(vkg_ctx *ctx, const float *d_hdr_rgba, uint32_t width, uint32_t height,
                                  const vkg_post_fx_settings *s, float *d_out_rgba, void *stream)
{
    if(!ctx) return VKG_ERR_INVALID_ARGUMENT;
    if(!s || ((width && height) && (!d_hdr_rgba || !d_out_rgba)))
        return set_error(ctx, VKG_ERR_INVALID_ARGUMENT, "vkg_post_fx: NULL argument");
    if(!(s->gamma > 0.f) || !std::isfinite(s->exposure) || !(s->brightness_thresh[1] > s->brightness_thresh[0]) ||
       s->blur_iterations > 64)
        return set_error(ctx, VKG_ERR_INVALID_ARGUMENT, "vkg_post_fx: invalid settings");
    if(width == 0 || height == 0) return VKG_OK;
    if(vkg_status st = bind_device(ctx); st != VKG_OK) return st;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const size_t n = (size_t)width * height;
    if(!s->tonemap)
    {
        // no post-FX: the HDR image itself (PBRPathTracer.cpp:411)
        VKG_TRY_CUDA(ctx, cudaMemcpyAsync(d_out_rgba, d_hdr_rgba, n * 4 * sizeof(float), cudaMemcpyDeviceToDevice, st));
        return VKG_OK;
    }
    // the 9-tap kernel, normalised in double (sigma from the size, see the file comment)
    blur_taps taps;
    {
        const double sigma = 0.3 * ((9 - 1) * 0.5 - 1) + 0.8;
        double sum = 0, k[9];
        for(int i = 0; i < 9; ++i)
        {
            const double x = i - 4;
            k[i] = std::exp(-x * x / (2 * sigma * sigma));
            sum += k[i];
        }
        for(int i = 0; i < 9; ++i) taps.w[i] = (float)(k[i] / sum);
    }
    const uint32_t bw = std::max<uint32_t>(width / 2, 1), bh = std::max<uint32_t>(height / 2, 1);
    __half *bl = nullptr;
    const __half *bloom = nullptr;
    if(s->bloom)
    {
        VKG_TRY_CUDA(ctx, ctx_alloc(ctx, reinterpret_cast<void **>(&bl), 2 * (size_t)bw * bh * 4 * sizeof(__half), st));
        __half *ping = bl, *pong = bl + (size_t)bw * bh * 4;
        // launches of up to three iterations; the first one thresholds
        const dim3 g((bw + BLOOM_TX - 1) / BLOOM_TX, (bh + BLOOM_TY - 1) / BLOOM_TY);
        uint32_t left = s->blur_iterations;
        const float4 *src = reinterpret_cast<const float4 *>(d_hdr_rgba);
        do
        {
            const uint32_t it = std::min(left, 3u);
            const size_t pixels = (size_t)(BLOOM_TX + 8 * it) * (BLOOM_TY + 8 * it);
            auto kern = it == 3 ? k_bloom<3> : it == 2 ? k_bloom<2> : it == 1 ? k_bloom<1> : k_bloom<0>;
            kern<<<g, BLOOM_THREADS, 2 * pixels * sizeof(uint2), st>>>(
                    src, width, height, s->brightness_thresh[0], s->brightness_thresh[1], ping, bw, bh, taps, pong);
            std::swap(ping, pong);
            src = nullptr;
            left -= it;
        } while(left);
        bloom = ping;
    }
    const dim3 blk(16, 16), g((width + 15) / 16, (height + 15) / 16);
    k_composite<<<g, blk, 0, st>>>(reinterpret_cast<const float4 *>(d_hdr_rgba), bloom, width, height, bw, bh,
                                   s->exposure, 1.f / s->gamma, reinterpret_cast<float4 *>(d_out_rgba));
    cudaError_t e = cudaGetLastError();
    if(bl)
    {
        const cudaError_t ef = cudaFreeAsync(bl, st);
        if(e == cudaSuccess) e = ef;
    }
    return e == cudaSuccess ? VKG_OK : cuda_check(ctx, e, "vkg_post_fx");
}
