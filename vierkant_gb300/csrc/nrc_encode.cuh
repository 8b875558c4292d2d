// Neural radiance cache: the input encoding shared by the mma.sync and tcgen05 kernels.
#pragma once

#include "nrc.cuh"

namespace vkg
{
namespace nrc
{

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi)
{
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t *>(&v);
}

// ---- encodings ---------------------------------------------------------------------------------
__device__ __forceinline__ void sh4(float x, float y, float z, float *o)
{
    // real spherical harmonics, bands 0..3
    const float xx = x * x, yy = y * y, zz = z * z;
    o[0] = 0.28209479177387814f;
    o[1] = -0.48860251190291987f * y;
    o[2] = 0.48860251190291987f * z;
    o[3] = -0.48860251190291987f * x;
    o[4] = 1.0925484305920792f * x * y;
    o[5] = -1.0925484305920792f * y * z;
    o[6] = 0.31539156525252005f * (3.f * zz - 1.f);
    o[7] = -1.0925484305920792f * x * z;
    o[8] = 0.5462742152960396f * (xx - yy);
    o[9] = -0.5900435899266435f * y * (3.f * xx - yy);
    o[10] = 2.890611442640554f * x * y * z;
    o[11] = -0.4570457994644658f * y * (5.f * zz - 1.f);
    o[12] = 0.3731763325901154f * z * (5.f * zz - 3.f);
    o[13] = -0.4570457994644658f * x * (5.f * zz - 1.f);
    o[14] = 1.445305721320277f * z * (xx - yy);
    o[15] = -0.5900435899266435f * x * (xx - 3.f * yy);
}

struct corner_iter
{
    uint32_t res, mask;
    bool dense;
    uint32_t cx, cy, cz;
    float fx, fy, fz;
};

__device__ __forceinline__ corner_iter level_setup(const grid_config &gc, uint32_t l, float px, float py, float pz)
{
    corner_iter c;
    c.res = gc.res[l];
    c.mask = (1u << gc.log2_t) - 1u;
    c.dense = (gc.dense >> l) & 1u;
    const float x = px * (float)c.res, y = py * (float)c.res, z = pz * (float)c.res;
    // the cell is clamped so p = 1 interpolates inside the last cell (every corner stays in range)
    const float top = (float)(c.res - 1);
    const float flx = fminf(floorf(x), top), fly = fminf(floorf(y), top), flz = fminf(floorf(z), top);
    c.cx = (uint32_t)(int)flx;
    c.cy = (uint32_t)(int)fly;
    c.cz = (uint32_t)(int)flz;
    c.fx = x - flx;
    c.fy = y - fly;
    c.fz = z - flz;
    return c;
}

// table entries and trilinear weights of the cell's corners; corner k is at x + (k & 1), y + (k >> 1 & 1),
// z + (k >> 2 & 1). Dense levels are indexed, the others hashed (x ^ y 2654435761 ^ z 805459861)
__device__ __forceinline__ void corners(const corner_iter &c, uint32_t (&idx)[8], float (&w)[8])
{
    if(c.dense)
    {
        const uint32_t s = c.res + 1, base = c.cx + (c.cy + c.cz * s) * s;
#pragma unroll
        for(int k = 0; k < 8; ++k) idx[k] = base + (k & 1) + ((k & 2) ? s : 0u) + ((k & 4) ? s * s : 0u);
    }
    else
    {
        const uint32_t hy = c.cy * 2654435761u, hz = c.cz * 805459861u;
#pragma unroll
        for(int k = 0; k < 8; ++k)
            idx[k] = ((c.cx + (k & 1)) ^ ((k & 2) ? hy + 2654435761u : hy) ^ ((k & 4) ? hz + 805459861u : hz)) & c.mask;
    }
#pragma unroll
    for(int k = 0; k < 8; ++k)
        w[k] = ((k & 1) ? c.fx : 1.f - c.fx) * ((k & 2) ? c.fy : 1.f - c.fy) * ((k & 4) ? c.fz : 1.f - c.fz);
}

__device__ __forceinline__ uint32_t quad_word(const uint4 &q, uint32_t i)
{
    const uint32_t a = (i & 1u) ? q.y : q.x, b = (i & 1u) ? q.w : q.z;
    return (i & 2u) ? b : a;
}

// v = *p if cond, as a predicated load (a branch per entry costs its reconvergence)
__device__ __forceinline__ void ld_if(uint32_t cond, const uint32_t *p, uint32_t &v)
{
    asm("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q ld.global.nc.u32 %0, [%1];\n}" : "+r"(v) : "l"(p), "r"(cond));
}

// BF16 feature pair of one level: the eight corners' entries interpolated. The gathers are bound by
// L1 lookups (one line a cycle and SM: 128 entries a record took 916 us for 2,073,600 records), so an
// entry is read with the aligned four that hold it: corners k and k + 1 of an x pair differ in the low
// bits of their index only (dense levels: by one), and lie in one four in three cases of four.
__device__ __forceinline__ uint32_t encode_level(const grid_config &gc, const __half2 *__restrict__ grid, uint32_t l,
                                                 float px, float py, float pz)
{
    const corner_iter c = level_setup(gc, l, px, py, pz);
    const uint32_t *tab = reinterpret_cast<const uint32_t *>(grid) + ((size_t)l << gc.log2_t);
    float w[8];
    uint32_t idx[8], e[8];
    uint4 q[4];
    corners(c, idx, w);
#pragma unroll
    for(int p = 0; p < 4; ++p) q[p] = __ldg(reinterpret_cast<const uint4 *>(tab) + (idx[2 * p] >> 2));
#pragma unroll
    for(int p = 0; p < 4; ++p)
    {
        e[2 * p] = quad_word(q[p], idx[2 * p]);
        e[2 * p + 1] = quad_word(q[p], idx[2 * p + 1]);
        ld_if((idx[2 * p] ^ idx[2 * p + 1]) >> 2, tab + idx[2 * p + 1], e[2 * p + 1]);
    }
    float f0 = 0.f, f1 = 0.f;
#pragma unroll
    for(int k = 0; k < 8; ++k)
    {
        const float2 v = __half22float2(*reinterpret_cast<const __half2 *>(&e[k]));
        f0 += w[k] * v.x;
        f1 += w[k] * v.y;
    }
    return pack_bf16(f0, f1);
}

__device__ __forceinline__ void normalised_pos(const grid_config &gc, const float *f, float &px, float &py, float &pz)
{
    px = fminf(fmaxf((f[0] - gc.smin[0]) * gc.sinv[0], 0.f), 1.f);
    py = fminf(fmaxf((f[1] - gc.smin[1]) * gc.sinv[1], 0.f), 1.f);
    pz = fminf(fmaxf((f[2] - gc.smin[2]) * gc.sinv[2], 0.f), 1.f);
}

// hash-grid features of levels [l0, l1) of one record: out[l - l0] = BF16 pair of level l
// (levels at or past gc.levels give zeros)
template<int L0, int L1>
__device__ __forceinline__ void encode_levels(const grid_config &gc, const __half2 *__restrict__ grid, float px,
                                              float py, float pz, uint32_t *out)
{
#pragma unroll
    for(int l = L0; l < L1; ++l) out[l - L0] = (uint32_t)l < gc.levels ? encode_level(gc, grid, l, px, py, pz) : 0u;
}

// the 16 SH coefficients of a direction as BF16 pairs
__device__ __forceinline__ void encode_sh(const float *d, uint32_t *out)
{
    float s[16];
    sh4(d[0], d[1], d[2], s);
#pragma unroll
    for(int k = 0; k < 8; ++k) out[k] = pack_bf16(s[2 * k], s[2 * k + 1]);
}

// the non-grid inputs (words 16..39): SH of the direction and of the normal, roughness, albedo, padding
__device__ __forceinline__ void encode_rest(const float *f, uint32_t *out)
{
    encode_sh(f + 3, out);
    encode_sh(f + 6, out + 8);
    out[16] = pack_bf16(f[9], f[10]);
    out[17] = pack_bf16(f[11], f[12]);
#pragma unroll
    for(int k = 18; k < 24; ++k) out[k] = 0u;
}

}// namespace nrc
}// namespace vkg
