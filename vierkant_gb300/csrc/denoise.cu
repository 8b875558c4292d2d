// Edge-avoiding a-trous denoiser over the path tracer's pixel records: the reference's denoise pass
// (src/PBRPathTracer.cpp:346-403, shaders/slang/denoise.slang) as CUDA kernels.
//
// Per pass (steps 1, 2, 4, 8, 16; PBRPathTracer.cpp:26) every pixel takes the 5x5 B3-spline kernel
// at offsets k * step (border-clamped) over albedo-demodulated radiance, each tap weighted by
//   exp(-(lum_c - lum_t)^2 / 0.9) * exp(-|n_c - n_t|^2 / 0.3) * exp(-|depth_c - depth_t|)
// (luminance of the demodulated colour with the NTSC weights, octahedral-decoded normals), and
// re-modulates with the centre's albedo clamped to >= 0.01. The three factors are evaluated as one
// exponential of the summed exponents (each factor is <= 1, so the reference's min(., 1) clamps are
// identities); pass k + 1 reads pass k's output.
//
// GB300 mapping: a stencil bound by issue and the latency of its loads (a 1280x720 frame's 15 MB of tap
// data a buffer stays in L2). One kernel decodes normals and depth into a float4, the clamped albedo into
// another and demodulates the radiance; then one kernel per pass. A thread filters DN_ROWS pixels of a
// column that lie `step` apart: their 5x5 taps fall on the same DN_ROWS + 4 rows, so a tap is loaded once
// for both, and a column's taps are loaded ahead of their use. It demodulates its own result for the
// next pass, which as a pass of its own took a launch and 32 bytes a pixel more. 1280x720: 226 -> 168 us
// (four rows a thread 167, 1920x1080 374 against 362, 400x300 55 against 48; taps loaded one at a time
// 173-188; two pixels packed in 64-bit FMAs 179).
#include "internal.hpp"
#include "pixel.cuh"

#include <cuda_runtime.h>

#include <utility>

namespace vkg
{
namespace
{

constexpr int DN_ROWS = 2; // pixels of a column per thread
constexpr uint32_t ATROUS_STEPS[5] = {1u, 2u, 4u, 8u, 16u};

// NTSC luminance weights (utils/color.slang:43)
constexpr float LUM_R = 0.298999994993f, LUM_G = 0.587000012398f, LUM_B = 0.114000000060f;

// a 16-byte load that stays where it is written (the compiler sinks __ldg to its use, which leaves the
// filter waiting on one tap at a time)
__device__ __forceinline__ float4 ld_nc(const float4 *p)
{
    float4 v;
    asm volatile("ld.global.nc.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}

// a colour divided by the clamped albedo, and its luminance
__device__ __forceinline__ float4 demodulate(float r, float g, float b, float4 a)
{
    r = r / a.x;
    g = g / a.y;
    b = b / a.z;
    return make_float4(r, g, b, r * LUM_R + g * LUM_G + b * LUM_B);
}

// per frame: (decoded normal, depth), (albedo clamped to >= 0.01, 0) and the demodulated radiance
__global__ void __launch_bounds__(256)
        k_dn_geometry(const vkg_pixel_data *__restrict__ px, uint32_t n, float4 *__restrict__ geo,
                      float4 *__restrict__ alb, float4 *__restrict__ dm, float *__restrict__ out_depth)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= n) return;
    const vkg_pixel_data p = px[i];
    const float2 q = unpack_snorm_2x16(p.normal);
    const float3 nv = oct_decode(q.x, q.y);
    geo[i] = make_float4(nv.x, nv.y, nv.z, p.depth);
    const float3 c = unpack_rgb8(p.albedo);
    const float4 a = make_float4(fmaxf(c.x, 0.01f), fmaxf(c.y, 0.01f), fmaxf(c.z, 0.01f), 0.f);
    alb[i] = a;
    dm[i] = demodulate(p.radiance[0], p.radiance[1], p.radiance[2], a);
    if(out_depth) out_depth[i] = p.depth;
}

// one a-trous pass: out = (sum_k w_k c_k / sum_k w_k) * albedo_centre, demodulated again unless LAST.
// Thread row g of the grid filters rows 2 step (g / step) + g mod step + {0, 1} step.
template<bool LAST>
__global__ void __launch_bounds__(128, 6)
        k_dn_filter(const float4 *__restrict__ dm, const float4 *__restrict__ geo, const float4 *__restrict__ alb,
                    uint32_t w, uint32_t h, int step, float4 *__restrict__ out)
{
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int g = (blockIdx.z * gridDim.y + blockIdx.y) * blockDim.y + threadIdx.y; // (grids are 65,535 blocks high at most)
    const int y0 = g / step * (DN_ROWS * step) + g % step;
    if(x >= (int)w || y0 >= (int)h) return;
    const float color_phi = 1.f / .9f, normal_phi = 1.f / .3f, position_phi = 1.f;
    float4 gc[DN_ROWS];
    float lc[DN_ROWS], sr[DN_ROWS], sg[DN_ROWS], sb[DN_ROWS], cw[DN_ROWS];
#pragma unroll
    for(int j = 0; j < DN_ROWS; ++j)
    {
        const uint32_t c = (uint32_t)min(y0 + j * step, (int)h - 1) * w + (uint32_t)x;
        gc[j] = __ldg(&geo[c]);
        lc[j] = __ldg(&dm[c]).w;
        sr[j] = sg[j] = sb[j] = cw[j] = 0.f;
    }
    uint32_t row[DN_ROWS + 4];
#pragma unroll
    for(int r = 0; r < DN_ROWS + 4; ++r) row[r] = (uint32_t)min(max(y0 + (r - 2) * step, 0), (int)h - 1) * w;
    // (the columns are a loop: unrolled as well, the code outgrows the instruction cache)
#pragma unroll 1
    for(int i = 0; i < 5; ++i)
    {
        const uint32_t ux = (uint32_t)min(max(x + (i - 2) * step, 0), (int)w - 1);
        const float bi = i == 2 ? 3.f / 8.f : (i & 1) ? 1.f / 4.f : 1.f / 16.f;
        const float kw[3] = {bi * (1.f / 16.f), bi * (1.f / 4.f), bi * (3.f / 8.f)};
        // the column's taps are all in flight before the first is used
        float4 d[DN_ROWS + 4], t[DN_ROWS + 4];
#pragma unroll
        for(int r = 0; r < DN_ROWS + 4; ++r)
        {
            d[r] = ld_nc(&dm[row[r] + ux]);
            t[r] = ld_nc(&geo[row[r] + ux]);
        }
#pragma unroll
        for(int r = 0; r < DN_ROWS + 4; ++r)
        {
            const float4 dt = d[r], gt = t[r];
#pragma unroll
            for(int j = 0; j < DN_ROWS; ++j)
            {
                const int k = r - j;
                if(k < 0 || k > 4) continue; // not a row of pixel j's kernel
                const float ld = lc[j] - dt.w;
                const float ex = gc[j].x - gt.x, ey = gc[j].y - gt.y, ez = gc[j].z - gt.z;
                const float e = ld * ld * color_phi + (ex * ex + ey * ey + ez * ez) * normal_phi +
                                fabsf(gc[j].w - gt.w) * position_phi;
                const float wk = expf(-e) * kw[k < 3 ? k : 4 - k];
                sr[j] += dt.x * wk;
                sg[j] += dt.y * wk;
                sb[j] += dt.z * wk;
                cw[j] += wk;
            }
        }
    }
#pragma unroll
    for(int j = 0; j < DN_ROWS; ++j)
    {
        const int y = y0 + j * step;
        if(y >= (int)h) break;
        const uint32_t c = (uint32_t)y * w + (uint32_t)x;
        const float4 a = __ldg(&alb[c]);
        const float r = sr[j] / cw[j] * a.x, gg = sg[j] / cw[j] * a.y, b = sb[j] / cw[j] * a.z;
        out[c] = LAST ? make_float4(r, gg, b, 0.f) : demodulate(r, gg, b, a);
    }
}

__global__ void k_dn_to_rgb(const float4 *__restrict__ in, uint32_t n, float *__restrict__ rgb)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= n) return;
    const float4 v = in[i];
    rgb[3 * (size_t)i] = v.x;
    rgb[3 * (size_t)i + 1] = v.y;
    rgb[3 * (size_t)i + 2] = v.z;
}

}// namespace

// the five passes; the result in rgba (stride 4) and / or rgb (stride 3)
vkg_status denoise_run(vkg_ctx *ctx, const vkg_pixel_data *px, uint32_t w, uint32_t h, float *out_rgba,
                       float *out_rgb, float *out_depth, cudaStream_t st)
{
    const size_t n = (size_t)w * h;
    if(n == 0) return VKG_OK;
    float4 *buf = nullptr;
    cudaError_t e = ctx_alloc(ctx, reinterpret_cast<void **>(&buf), 4 * n * sizeof(float4), st);
    if(e != cudaSuccess) return cuda_check(ctx, e, "vkg_denoise scratch");
    float4 *geo = buf, *alb = buf + n, *ping = buf + 2 * n, *pong = buf + 3 * n;
    const uint32_t g1 = (uint32_t)((n + 255) / 256);
    k_dn_geometry<<<g1, 256, 0, st>>>(px, (uint32_t)n, geo, alb, ping, out_depth);
    const dim3 blk(32, 4);
    for(int pass = 0; pass < 5; ++pass)
    {
        const uint32_t step = ATROUS_STEPS[pass], groups = (h + DN_ROWS * step - 1) / (DN_ROWS * step) * step;
        const uint32_t rows = (groups + blk.y - 1) / blk.y, layers = (rows + 65534u) / 65535u;
        const dim3 grid((w + blk.x - 1) / blk.x, (rows + layers - 1) / layers, layers);
        if(pass + 1 < 5)
            k_dn_filter<false><<<grid, blk, 0, st>>>(ping, geo, alb, w, h, (int)step, pong);
        else
            k_dn_filter<true><<<grid, blk, 0, st>>>(ping, geo, alb, w, h, (int)step,
                                                    out_rgba ? reinterpret_cast<float4 *>(out_rgba) : pong);
        std::swap(ping, pong);
    }
    const float4 *prev = out_rgba ? reinterpret_cast<const float4 *>(out_rgba) : ping;
    if(out_rgb) k_dn_to_rgb<<<g1, 256, 0, st>>>(prev, (uint32_t)n, out_rgb);
    e = cudaGetLastError();
    const cudaError_t ef = cudaFreeAsync(buf, st);
    if(e == cudaSuccess) e = ef;
    return e == cudaSuccess ? VKG_OK : cuda_check(ctx, e, "vkg_denoise");
}

}// namespace vkg

using namespace vkg;

extern "C" vkg_status vkg_denoise(vkg_ctx *ctx, const vkg_pixel_data *d_pixels, uint32_t width, uint32_t height,
                                  float *d_out_rgba, float *d_out_depth, void *stream)
{
    if(!ctx) return VKG_ERR_INVALID_ARGUMENT;
    if((width && height) && (!d_pixels || !d_out_rgba))
        return set_error(ctx, VKG_ERR_INVALID_ARGUMENT, "vkg_denoise: NULL buffer");
    if(vkg_status s = bind_device(ctx); s != VKG_OK) return s;
    return denoise_run(ctx, d_pixels, width, height, d_out_rgba, nullptr, d_out_depth,
                       static_cast<cudaStream_t>(stream));
}
