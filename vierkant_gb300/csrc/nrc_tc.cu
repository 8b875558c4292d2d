// Neural radiance cache inference on the 5th-generation tensor cores (tcgen05, sm_103a).
//
// One CTA of 256 threads owns a tile of 128 queries at a time (persistent over tiles):
//   1. two threads per query encode it (hash-grid levels 0..7 / levels 8..15 + SH + material,
//      nrc_encode.cuh) straight into shared memory as the BF16 A operand of layer 0 (128 x 80,
//      canonical K-major layout, tc.cuh);
//   2. thread 0 issues the layer's tcgen05.mma steps (M = 128, N = 64 or 16, K = 16 each) against
//      the weights, which stay in shared memory for the kernel's lifetime, and commits them to an
//      mbarrier; the FP32 accumulator lives in TMEM (64 columns);
//   3. after the mbarrier (bounded wait), the two threads of a query read its TMEM lane (32 columns
//      each), apply ReLU, pack BF16 and write the next layer's A operand back to shared memory; the
//      last layer's first three columns are the prediction.
// The numerics equal the mma.sync twin (nrc.cu): BF16 inputs / weights / activations, FP32
// accumulation; only the summation order inside an MMA differs.
//
// A wait that runs out (it never should) sets bit 0 of the error word, lets any MMA still in flight
// finish (bounded), frees the TMEM and returns.
#include "nrc_encode.cuh"
#include "tc.cuh"

#include <algorithm>

namespace vkg
{
namespace nrc
{

constexpr uint32_t TC_THREADS = 128, TC_INFER_THREADS = 256, TC_TILE = 128, TC_TMEM_COLS = 64;
constexpr uint32_t TC_W_BYTES = NPARAM * 2;      // all six layers, BF16 B operands (45,056 B)
constexpr uint32_t TC_A_BYTES = TC_TILE * IN * 2; // one A operand (20,480 B)
constexpr uint32_t TC_SMEM = TC_W_BYTES + TC_A_BYTES;
constexpr uint32_t TC_TIMEOUT = 1u;

namespace
{

__device__ __forceinline__ uint32_t eff_n(uint32_t n, const uint32_t *d_n) { return d_n ? min(*d_n, n) : n; }

// encodes the feature records of a tile and runs them through the MLP
__global__ void __launch_bounds__(TC_INFER_THREADS)
        k_infer_tc(const float *__restrict__ feats, uint32_t n_cap, const uint32_t *__restrict__ d_n, grid_config gc,
                   const __half2 *__restrict__ grid, const uint16_t *__restrict__ wtc, float *__restrict__ Y,
                   uint32_t *__restrict__ err)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t mbar;
    __shared__ uint32_t tslot;
    uint8_t *sw = smem, *sa = smem + TC_W_BYTES;
    const uint32_t tid = threadIdx.x, warp = tid >> 5;
    // thread t works on row r = t mod 128 of the tile; its half h = t / 128 picks the hash-grid levels
    // it encodes (0..7 or 8..15 + the SH / material inputs) and the TMEM columns it drains (warp w reads
    // TMEM lanes 32 (w mod 4) .. + 31)
    const uint32_t r = tid & (TC_TILE - 1), h = tid >> 7;

    for(uint32_t i = tid; i < TC_W_BYTES / 16; i += TC_INFER_THREADS)
        reinterpret_cast<uint4 *>(sw)[i] = reinterpret_cast<const uint4 *>(wtc)[i];
    if(warp == 0) tc::tmem_alloc(&tslot, TC_TMEM_COLS);
    if(tid == 0) tc::mbar_init(&mbar, 1);
    tc::fence_async_smem();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tslot, lane_base = ((warp & 3u) * 32u) << 16;
    const uint32_t sw_addr = tc::smem_addr(sw), sa_addr = tc::smem_addr(sa);
    const uint32_t n = eff_n(n_cap, d_n), tiles = (n + TC_TILE - 1) / TC_TILE;
    uint32_t phase = 0;
    bool failed = false;

    for(uint32_t tile = blockIdx.x; tile < tiles && !failed; tile += gridDim.x)
    {
        const uint32_t q = tile * TC_TILE + r;
        if(h == 0)
        {
            uint32_t x[8];
            if(q < n)
            {
                const float *f = feats + (size_t)FEAT * q;
                float px, py, pz;
                normalised_pos(gc, f, px, py, pz);
                encode_levels<0, 8>(gc, grid, px, py, pz, x);
            }
            else
                for(int j = 0; j < 8; ++j) x[j] = 0u;
#pragma unroll
            for(int j = 0; j < 2; ++j)
                *reinterpret_cast<uint4 *>(sa + tc::canon_offset(r, 8 * j, IN)) =
                        make_uint4(x[4 * j], x[4 * j + 1], x[4 * j + 2], x[4 * j + 3]);
        }
        else
        {
            uint32_t x[32];
            if(q < n)
            {
                const float *f = feats + (size_t)FEAT * q;
                float px, py, pz;
                normalised_pos(gc, f, px, py, pz);
                encode_levels<8, 16>(gc, grid, px, py, pz, x);
                encode_rest(f, x + 8);
            }
            else
                for(int j = 0; j < 32; ++j) x[j] = 0u;
#pragma unroll
            for(int j = 0; j < 8; ++j)
                *reinterpret_cast<uint4 *>(sa + tc::canon_offset(r, 16 + 8 * j, IN)) =
                        make_uint4(x[4 * j], x[4 * j + 1], x[4 * j + 2], x[4 * j + 3]);
        }
        tc::fence_async_smem();
        tc::fence_before_sync();
        __syncthreads();
#pragma unroll 1
        for(int l = 0; l < NLAYER; ++l)
        {
            const uint32_t K = layer_in(l), N = layer_out(l);
            if(tid == 0)
            {
                tc::fence_after_sync();
                const uint32_t idesc = tc::idesc_bf16(TC_TILE, N);
                const uint32_t wb = sw_addr + (uint32_t)layer_off(l) * 2u;
                for(uint32_t s = 0; s < K / 16; ++s)
                    tc::mma_bf16(tmem, tc::smem_desc(sa_addr + 256u * s, 128u, K * 16u),
                                 tc::smem_desc(wb + 256u * s, 128u, K * 16u), idesc, s > 0);
                tc::mma_commit(&mbar);
            }
            const bool ok = tc::mbar_wait(&mbar, phase);
            if(__syncthreads_or(!ok))
            {
                failed = true;
                break;
            }
            phase ^= 1u;
            tc::fence_after_sync();
            if(l + 1 < NLAYER)
            {
                // this thread's 32 of the 64 columns of row r
                uint32_t hv[16];
#pragma unroll
                for(int c = 0; c < 2; ++c)
                {
                    float v[16];
                    tc::tmem_ld16(tmem + lane_base + 32u * h + 16u * c, v);
                    tc::tmem_ld_wait();
#pragma unroll
                    for(int j = 0; j < 8; ++j) hv[8 * c + j] = pack_bf16(fmaxf(v[2 * j], 0.f), fmaxf(v[2 * j + 1], 0.f));
                }
#pragma unroll
                for(int j = 0; j < 4; ++j)
                    *reinterpret_cast<uint4 *>(sa + tc::canon_offset(r, 32 * h + 8 * j, HID)) =
                            make_uint4(hv[4 * j], hv[4 * j + 1], hv[4 * j + 2], hv[4 * j + 3]);
                tc::fence_async_smem();
            }
            else if(h == 0)
            {
                float v[16];
                tc::tmem_ld16(tmem + lane_base, v);
                tc::tmem_ld_wait();
                if(q < n)
                {
                    Y[3 * (size_t)q] = v[0];
                    Y[3 * (size_t)q + 1] = v[1];
                    Y[3 * (size_t)q + 2] = v[2];
                }
            }
            tc::fence_before_sync();
            __syncthreads();
        }
    }
    if(failed)
    {
        if(tid == 0) atomicOr(err, TC_TIMEOUT);
        tc::mbar_wait(&mbar, phase); // the MMAs in flight, if any
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if(warp == 0) tc::tmem_dealloc(tmem, TC_TMEM_COLS);
}

// diagnostic: D (128 x N, FP32) = A (128 x K BF16, row-major) * B^T (N x K BF16, row-major) through the
// same descriptors, one CTA
__global__ void __launch_bounds__(TC_THREADS)
        k_tc_gemm(const uint16_t *__restrict__ A, const uint16_t *__restrict__ B, uint32_t K, uint32_t N,
                  float *__restrict__ D, uint32_t *__restrict__ err)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t mbar;
    __shared__ uint32_t tslot;
    const uint32_t tid = threadIdx.x, warp = tid >> 5;
    uint8_t *sa = smem, *sb = smem + TC_TILE * K * 2;
    for(uint32_t k = 0; k < K; ++k)
        *reinterpret_cast<uint16_t *>(sa + tc::canon_offset(tid, k, K)) = A[(size_t)tid * K + k];
    for(uint32_t e = tid; e < N * K; e += TC_THREADS)
        *reinterpret_cast<uint16_t *>(sb + tc::canon_offset(e / K, e % K, K)) = B[e];
    if(warp == 0) tc::tmem_alloc(&tslot, TC_TMEM_COLS);
    if(tid == 0) tc::mbar_init(&mbar, 1);
    tc::fence_async_smem();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tslot;
    if(tid == 0)
    {
        const uint32_t idesc = tc::idesc_bf16(TC_TILE, N);
        for(uint32_t s = 0; s < K / 16; ++s)
            tc::mma_bf16(tmem, tc::smem_desc(tc::smem_addr(sa) + 256u * s, 128u, K * 16u),
                         tc::smem_desc(tc::smem_addr(sb) + 256u * s, 128u, K * 16u), idesc, s > 0);
        tc::mma_commit(&mbar);
    }
    const bool ok = tc::mbar_wait(&mbar, 0);
    if(__syncthreads_or(!ok))
    {
        if(tid == 0) atomicOr(err, TC_TIMEOUT);
        tc::mbar_wait(&mbar, 0);
    }
    else
    {
        tc::fence_after_sync();
        for(uint32_t c = 0; c < N / 16; ++c)
        {
            float v[16];
            tc::tmem_ld16(tmem + ((warp * 32u) << 16) + 16u * c, v);
            tc::tmem_ld_wait();
            for(int j = 0; j < 16; ++j) D[(size_t)tid * N + 16 * c + j] = v[j];
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if(warp == 0) tc::tmem_dealloc(tmem, TC_TMEM_COLS);
}

// ---- pipelined inference: independent warpgroups ------------------------------------------------
// The single-tile kernel above leaves the tensor core idle while a layer's epilogue runs, and the
// epilogue, not the MMA, sets its time. Here a CTA of NWG warpgroups (128 threads each) runs NWG tiles
// at once, each with 96 TMEM columns, an mbarrier and a named barrier of its own, and its thread 0
// issues its own MMAs; so while one warpgroup drains its accumulator the tensor core works on
// another's layer. The weights (all six layers, 45 KB) are shared. Thread r of a warpgroup owns row r of
// its tile (TMEM lane r: warp w reads lanes 32 (w mod 4) .. + 31).
// Layer 0 reads the encoded BF16 records of k_encode from shared memory (canonical K-major), copied there
// by cp.async while the tile before runs its later layers. The hidden layers read their operand from
// TMEM: the epilogue (64 columns in, ReLU, BF16) stores 32 columns back with tcgen05.st, which takes the
// 16 KB a layer and tile of shared-memory stores and reads out of the way. 2,073,600 queries: 222 us
// with operands in shared memory and eight warpgroups, 183 us with four this way.
// TMEM columns a CTA of g warpgroups allocates when each uses `per`: a power of two of at least 32
__host__ __device__ constexpr uint32_t tmem_columns(uint32_t per, uint32_t g)
{
    uint32_t c = 32;
    while(c < per * g) c *= 2;
    return c;
}
constexpr uint32_t TC_WG_COLS = 96; // per warpgroup: 64 of the accumulator, 32 of the next layer's operand

template<int NWG>
__global__ void __launch_bounds__(NWG * 128)
        k_infer_tc_wg(const uint32_t *__restrict__ X, uint32_t n_cap, const uint32_t *__restrict__ d_n,
                      const uint16_t *__restrict__ wtc, float *__restrict__ Y, uint32_t *__restrict__ err)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t mbar[NWG];
    __shared__ uint32_t tslot;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, g = tid >> 7, r = tid & 127u;
    uint8_t *sw = smem, *sa = smem + TC_W_BYTES + g * TC_A_BYTES;
    const uint32_t sw_addr = tc::smem_addr(sw), sa_addr = tc::smem_addr(sa);
    const uint32_t n = eff_n(n_cap, d_n), tiles = (n + TC_TILE - 1) / TC_TILE;
    // this thread's row of a tile's layer-0 operand (zeros past n)
    auto load = [&](uint32_t tile) {
        const uint32_t q = tile * TC_TILE + r;
        const uint32_t *src = X + (size_t)(IN / 2) * (q < n ? q : 0u);
#pragma unroll
        for(int j = 0; j < IN / 8; ++j)
            tc::cp_async16(sa_addr + tc::canon_offset(r, 8 * j, IN), src + 4 * j, q < n);
    };
    const uint32_t first = blockIdx.x * NWG + g;
    if(first < tiles) load(first);
    for(uint32_t i = tid; i < TC_W_BYTES / 16; i += NWG * 128)
        tc::cp_async16(sw_addr + 16u * i, reinterpret_cast<const uint4 *>(wtc) + i, true);
    static_assert(NWG >= 1 && NWG * TC_WG_COLS <= 512, "at most 512 TMEM columns");
    constexpr uint32_t COLS = tmem_columns(TC_WG_COLS, NWG);
    if(warp == 0) tc::tmem_alloc(&tslot, COLS);
    if(tid < NWG) tc::mbar_init(&mbar[tid], 1);
    tc::cp_async_commit();
    tc::cp_async_wait<0>();
    tc::fence_async_smem();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tslot + TC_WG_COLS * g, ta = tmem + 64u, lane_base = ((warp & 3u) * 32u) << 16;
    const uint32_t bar_id = g + 1;
    uint32_t phase = 0;
    bool failed = false;

    for(uint32_t tile = first; tile < tiles && !failed; tile += gridDim.x * NWG)
    {
        const uint32_t q = tile * TC_TILE + r;
        // the tile's rows were loaded during the tile before
        tc::cp_async_wait<0>();
        tc::fence_async_smem();
        tc::fence_before_sync();
        tc::wg_sync(bar_id);
#pragma unroll 1
        for(int l = 0; l < NLAYER; ++l)
        {
            const uint32_t K = layer_in(l), N = layer_out(l);
            if(r == 0)
            {
                tc::fence_after_sync();
                const uint32_t idesc = tc::idesc_bf16(TC_TILE, N);
                const uint32_t wb = sw_addr + (uint32_t)layer_off(l) * 2u;
                for(uint32_t s = 0; s < K / 16; ++s)
                {
                    const uint64_t b = tc::smem_desc(wb + 256u * s, 128u, K * 16u);
                    if(l == 0) tc::mma_bf16(tmem, tc::smem_desc(sa_addr + 256u * s, 128u, K * 16u), b, idesc, s > 0);
                    else tc::mma_bf16_ts(tmem, ta + 8u * s, b, idesc, s > 0);
                }
                tc::mma_commit(&mbar[g]);
            }
            const bool ok = tc::mbar_wait(&mbar[g], phase);
            if(tc::wg_sync_or(bar_id, !ok))
            {
                failed = true;
                break;
            }
            phase ^= 1u;
            tc::fence_after_sync();
            if(l == 0 && tile + gridDim.x * NWG < tiles)
            {
                load(tile + gridDim.x * NWG); // layer 0 is done with the operand
                tc::cp_async_commit();
            }
            if(l + 1 < NLAYER)
            {
                // two TMEM loads in flight per wait
#pragma unroll
                for(int c2 = 0; c2 < 2; ++c2)
                {
                    float v[2][16];
                    tc::tmem_ld16(tmem + lane_base + 32u * c2, v[0]);
                    tc::tmem_ld16(tmem + lane_base + 32u * c2 + 16u, v[1]);
                    tc::tmem_ld_wait();
                    uint32_t hv[16];
#pragma unroll
                    for(int j = 0; j < 16; ++j)
                        hv[j] = pack_bf16(fmaxf(v[j >> 3][2 * (j & 7)], 0.f), fmaxf(v[j >> 3][2 * (j & 7) + 1], 0.f));
                    tc::tmem_st16(ta + lane_base + 16u * c2, hv);
                }
                tc::tmem_st_wait();
            }
            else
            {
                float v[16];
                tc::tmem_ld16(tmem + lane_base, v);
                tc::tmem_ld_wait();
                if(q < n)
                {
                    Y[3 * (size_t)q] = v[0];
                    Y[3 * (size_t)q + 1] = v[1];
                    Y[3 * (size_t)q + 2] = v[2];
                }
            }
            tc::fence_before_sync();
            tc::wg_sync(bar_id);
        }
    }
    tc::cp_async_wait<0>();
    if(failed)
    {
        if(r == 0) atomicOr(err, TC_TIMEOUT);
        tc::mbar_wait(&mbar[g], phase); // this warpgroup's MMAs in flight, if any
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if(warp == 0) tc::tmem_dealloc(tslot, COLS);
}

// ---- training forward and backward on tcgen05 ---------------------------------------------------
// The mma.sync k_forward<true> and k_backward as one pass over the tiles, with the warpgroup pipeline of
// k_infer_tc_wg: per tile of 128 records, thread r owns record q = 128 tile + r:
//   forward as in k_infer_tc_wg; H_1..H_5 go to memory for the weight gradients, and one bit an
//   activation, H > 0, stays in registers;
//   dy = dL/dy of the relative L2 loss (|y - t|^2 / (y^2 + 0.01), mean over 3n) -> G block 5 and the
//   BF16 A operand (128 x 16, shared memory);
//   for l = 5 .. 1: D = G_l W_l^T (UMMA, TMEM), G_{l-1} = D * [H_l > 0] rounded to BF16 -> G block
//   l - 1 and the next A operand (128 x 64), in TMEM as in the forward;
//   dX (the 32 hash-grid features) = G_0 W_0^T (N = 32) -> dXg in FP32.
// Quantisation points equal the mma.sync kernels' (FP32 sums, BF16 rounding of each H and G); only the
// summation order inside an MMA differs. Both weight layouts (wtc, and wtc_t transposed) are resident.
// H, G and dXg are stored by tiles: 16-byte group p of a record's P groups at group (tile P + p) 128 + r,
// so that a warp's stores are whole lines (by records each 16-byte store touched 32).
// Bound by the chain of twelve layers and its stores (1.4 KB a record, to L2): 65,536 records in 25 us; as two
// kernels with the records' rows, the activations read back, 56 us.
constexpr uint32_t TC_G_BYTES = TC_TILE * OUTP * 2; // the backward's first A operand (4,096 B)
template<int NWG>
__global__ void __launch_bounds__(NWG * 128)
        k_train_tc_wg(const uint32_t *__restrict__ X, const float *__restrict__ T, uint32_t n_cap,
                      const uint32_t *__restrict__ d_n, const uint16_t *__restrict__ wtc,
                      const uint16_t *__restrict__ wtc_t, uint4 *__restrict__ H, uint4 *__restrict__ G,
                      float4 *__restrict__ dXg, float *__restrict__ loss_sum, uint32_t *__restrict__ err)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t mbar[NWG];
    __shared__ uint32_t tslot;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, g = tid >> 7, r = tid & 127u;
    uint8_t *sg = smem + 2 * TC_W_BYTES + NWG * TC_A_BYTES + g * TC_G_BYTES;
    const uint32_t sw_addr = tc::smem_addr(smem), sa_addr = sw_addr + 2 * TC_W_BYTES + g * TC_A_BYTES;
    const uint32_t sg_addr = tc::smem_addr(sg);
    const uint32_t n = eff_n(n_cap, d_n), tiles = (n + TC_TILE - 1) / TC_TILE;
    // this thread's row of a tile's layer-0 operand (zeros past n)
    auto load = [&](uint32_t tile) {
        const uint32_t q = tile * TC_TILE + r;
        const uint32_t *src = X + (size_t)(IN / 2) * (q < n ? q : 0u);
#pragma unroll
        for(int j = 0; j < IN / 8; ++j)
            tc::cp_async16(sa_addr + tc::canon_offset(r, 8 * j, IN), src + 4 * j, q < n);
    };
    const uint32_t first = blockIdx.x * NWG + g;
    if(first < tiles) load(first);
    for(uint32_t i = tid; i < TC_W_BYTES / 16; i += NWG * 128)
    {
        tc::cp_async16(sw_addr + 16u * i, reinterpret_cast<const uint4 *>(wtc) + i, true);
        tc::cp_async16(sw_addr + TC_W_BYTES + 16u * i, reinterpret_cast<const uint4 *>(wtc_t) + i, true);
    }
    static_assert(NWG >= 1 && NWG * TC_WG_COLS <= 512, "at most 512 TMEM columns");
    constexpr uint32_t COLS = tmem_columns(TC_WG_COLS, NWG);
    if(warp == 0) tc::tmem_alloc(&tslot, COLS);
    if(tid < NWG) tc::mbar_init(&mbar[tid], 1);
    tc::cp_async_commit();
    tc::cp_async_wait<0>();
    tc::fence_async_smem();
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tslot + TC_WG_COLS * g, ta = tmem + 64u, lane_base = ((warp & 3u) * 32u) << 16;
    const float inv_count = n ? 1.f / (3.f * (float)n) : 0.f;
    const uint32_t bar_id = g + 1;
    uint32_t phase = 0;
    bool failed = false;
    float loss = 0.f;

    // D (128 x rows) = A (128 x K) * B^T, the A operand in shared memory (at a, else 0) or TMEM; false if the
    // wait ran out
    auto multiply = [&](uint32_t a, uint32_t b, uint32_t K, uint32_t rows) {
        if(r == 0)
        {
            tc::fence_after_sync();
            const uint32_t idesc = tc::idesc_bf16(TC_TILE, rows);
            for(uint32_t s = 0; s < K / 16; ++s)
            {
                const uint64_t bd = tc::smem_desc(b + 256u * s, 128u, K * 16u);
                if(a) tc::mma_bf16(tmem, tc::smem_desc(a + 256u * s, 128u, K * 16u), bd, idesc, s > 0);
                else tc::mma_bf16_ts(tmem, ta + 8u * s, bd, idesc, s > 0);
            }
            tc::mma_commit(&mbar[g]);
        }
        const bool ok = tc::mbar_wait(&mbar[g], phase);
        if(tc::wg_sync_or(bar_id, !ok)) return false;
        phase ^= 1u;
        tc::fence_after_sync();
        return true;
    };

    for(uint32_t tile = first; tile < tiles && !failed; tile += gridDim.x * NWG)
    {
        const uint32_t q = tile * TC_TILE + r;
        const bool valid = q < n;
        float t[3] = {0.f, 0.f, 0.f}, y[3] = {0.f, 0.f, 0.f};
        if(valid)
            for(int c = 0; c < 3; ++c) t[c] = T[(size_t)q * 3 + c];
        uint4 *hp = H + tiled_group(q, ACT / 8, 0), *gp = G + tiled_group(q, GRAD / 8, 0);
        // H_l > 0 of the last layers first: bits j and 16 + j of word c are columns 32 c + 2 j and 32 c + 2 j + 1
        uint32_t pos[NLAYER - 1][2];
        // the tile's rows were loaded during the tile before
        tc::cp_async_wait<0>();
        tc::fence_async_smem();
        tc::fence_before_sync();
        tc::wg_sync(bar_id);
#pragma unroll 1
        for(int l = 0; l < NLAYER; ++l)
        {
            if(!multiply(l == 0 ? sa_addr : 0u, sw_addr + (uint32_t)layer_off(l) * 2u, layer_in(l), layer_out(l)))
            {
                failed = true;
                break;
            }
            if(l == 0 && tile + gridDim.x * NWG < tiles)
            {
                load(tile + gridDim.x * NWG); // layer 0 is done with the operand
                tc::cp_async_commit();
            }
            if(l + 1 < NLAYER)
            {
#pragma unroll
                for(int i = NLAYER - 2; i > 0; --i)
                {
                    pos[i][0] = pos[i - 1][0];
                    pos[i][1] = pos[i - 1][1];
                }
#pragma unroll
                for(int c = 0; c < 2; ++c)
                {
                    // two TMEM loads in flight per wait
                    float v[2][16];
                    tc::tmem_ld16(tmem + lane_base + 32u * c, v[0]);
                    tc::tmem_ld16(tmem + lane_base + 32u * c + 16u, v[1]);
                    tc::tmem_ld_wait();
                    uint32_t hv[16], bits = 0;
#pragma unroll
                    for(int j = 0; j < 16; ++j)
                    {
                        hv[j] = pack_bf16(fmaxf(v[j >> 3][2 * (j & 7)], 0.f), fmaxf(v[j >> 3][2 * (j & 7) + 1], 0.f));
                        // the sum carries into a half's top bit unless its value is zero
                        bits = (bits >> 1) | (((hv[j] & 0x7FFF7FFFu) + 0x7FFF7FFFu) & 0x80008000u);
                    }
                    pos[0][c] = bits;
                    tc::tmem_st16(ta + lane_base + 16u * c, hv);
                    if(valid)
#pragma unroll
                        for(int j = 0; j < 4; ++j)
                            hp[(8 * l + 4 * c + j) * TC_TILE] = make_uint4(hv[4 * j], hv[4 * j + 1], hv[4 * j + 2], hv[4 * j + 3]);
                }
                tc::tmem_st_wait();
                tc::fence_before_sync();
                tc::wg_sync(bar_id);
            }
            else
            {
                float v[16];
                tc::tmem_ld16(tmem + lane_base, v);
                tc::tmem_ld_wait();
                for(int c = 0; c < 3; ++c) y[c] = v[c];
            }
        }
        if(failed) break;
        // dL/dy (raw columns 0..2 of 16)
        float dy[3] = {0.f, 0.f, 0.f};
        if(valid)
            for(int c = 0; c < 3; ++c)
            {
                const float den = y[c] * y[c] + 0.01f;
                const float e = y[c] - t[c];
                loss += e * e / den;
                dy[c] = 2.f * e / den * inv_count;
            }
        const uint4 gy = make_uint4(pack_bf16(dy[0], dy[1]), pack_bf16(dy[2], 0.f), 0u, 0u), zero = make_uint4(0u, 0u, 0u, 0u);
        if(valid)
        {
            gp[8 * (NLAYER - 1) * TC_TILE] = gy;
            gp[(8 * (NLAYER - 1) + 1) * TC_TILE] = zero;
        }
        // A operand 128 x 16 (K = 16): columns 0..7 and 8..15
        *reinterpret_cast<uint4 *>(sg + tc::canon_offset(r, 0, 16)) = gy;
        *reinterpret_cast<uint4 *>(sg + tc::canon_offset(r, 8, 16)) = zero;
        tc::fence_async_smem();
        tc::fence_before_sync();
        tc::wg_sync(bar_id);
#pragma unroll 1
        for(int l = NLAYER - 1; l >= 0; --l)
        {
            // B = W_l as rows = inputs, K = outputs
            if(!multiply(l == NLAYER - 1 ? sg_addr : 0u, sw_addr + TC_W_BYTES + (uint32_t)layer_off(l) * 2u, layer_out(l),
                         l == 0 ? 32u : (uint32_t)layer_in(l)))
            {
                failed = true;
                break;
            }
            if(l > 0)
            {
                // G_{l-1} = dH_l * [H_l > 0]
#pragma unroll
                for(int c = 0; c < 2; ++c)
                {
                    float v[2][16];
                    tc::tmem_ld16(tmem + lane_base + 32u * c, v[0]);
                    tc::tmem_ld16(tmem + lane_base + 32u * c + 16u, v[1]);
                    tc::tmem_ld_wait();
                    uint32_t gv[16];
#pragma unroll
                    for(int j = 0; j < 16; ++j)
                        gv[j] = pack_bf16(v[j >> 3][2 * (j & 7)], v[j >> 3][2 * (j & 7) + 1]) &
                                (((pos[0][c] >> j) & 0x00010001u) * 0xFFFFu);
                    tc::tmem_st16(ta + lane_base + 16u * c, gv);
                    if(valid)
#pragma unroll
                        for(int j = 0; j < 4; ++j)
                            gp[(8 * (l - 1) + 4 * c + j) * TC_TILE] = make_uint4(gv[4 * j], gv[4 * j + 1], gv[4 * j + 2], gv[4 * j + 3]);
                }
#pragma unroll
                for(int i = 0; i < NLAYER - 2; ++i)
                {
                    pos[i][0] = pos[i + 1][0];
                    pos[i][1] = pos[i + 1][1];
                }
                tc::tmem_st_wait();
            }
            else
            {
                // dX of the 32 hash-grid features, FP32
                float4 *dp = dXg + tiled_group(q, 8, 0);
#pragma unroll
                for(int c = 0; c < 2; ++c)
                {
                    float v[16];
                    tc::tmem_ld16(tmem + lane_base + 16u * c, v);
                    tc::tmem_ld_wait();
                    if(valid)
#pragma unroll
                        for(int j = 0; j < 4; ++j)
                            dp[(4 * c + j) * TC_TILE] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
                }
            }
            tc::fence_before_sync();
            tc::wg_sync(bar_id);
        }
    }
    tc::cp_async_wait<0>();
    for(int o = 16; o > 0; o >>= 1) loss += __shfl_down_sync(0xffffffffu, loss, o);
    if((tid & 31u) == 0 && loss_sum) atomicAdd(loss_sum, loss * inv_count);
    if(failed)
    {
        if(r == 0) atomicOr(err, TC_TIMEOUT);
        tc::mbar_wait(&mbar[g], phase); // this warpgroup's MMAs in flight, if any
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if(warp == 0) tc::tmem_dealloc(tslot, COLS);
}

// diagnostic: the error path every tcgen05 kernel here takes when a wait runs out, run to its end on
// purpose. Each CTA allocates TMEM and waits on an mbarrier that nothing arrives on, with a limit of
// limit_ns instead of the kernels' 1 s; the wait gives up, the CTA sets TC_TIMEOUT, waits a second
// time (bounded, as the kernels do for MMAs in flight), frees its TMEM and returns. elapsed_ns: the
// longest time one CTA spent in the two waits.
constexpr uint32_t PROBE_TMEM_COLS = 32;
__global__ void __launch_bounds__(TC_THREADS)
        k_wait_probe(uint64_t limit_ns, uint32_t *__restrict__ err, unsigned long long *__restrict__ elapsed_ns)
{
    __shared__ uint64_t mbar;
    __shared__ uint32_t tslot;
    const uint32_t tid = threadIdx.x, warp = tid >> 5;
    if(warp == 0) tc::tmem_alloc(&tslot, PROBE_TMEM_COLS);
    if(tid == 0) tc::mbar_init(&mbar, 1);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tslot;
    const uint64_t t0 = tc::global_ns();
    const bool ok = tc::mbar_wait_for(&mbar, 0, tc::WAIT_LIMIT, limit_ns);
    if(__syncthreads_or(!ok))
    {
        if(tid == 0) atomicOr(err, TC_TIMEOUT);
        tc::mbar_wait_for(&mbar, 0, tc::WAIT_LIMIT, limit_ns);
    }
    if(tid == 0) atomicMax(elapsed_ns, (unsigned long long)(tc::global_ns() - t0));
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if(warp == 0) tc::tmem_dealloc(tmem, PROBE_TMEM_COLS);
}

// ---- weight gradients on tcgen05 --------------------------------------------------------------
// dW_l[k][o] = sum over records s of H_l[s][k] * G_l[s][o] (H_0 = the encoded inputs X, G_l the
// gradient of layer l's pre-activation, both BF16 as the backward stored them). As one UMMA chain per
// layer and chunk of 64 records: D (128 x N_l, FP32 in TMEM) += A (128 x 64) * B (N_l x 64)^T with
// A = H_l^T and B = G_l^T. A record's features are contiguous, so both operands are MN-major: a core
// matrix is 8 records x 8 features (16 bytes a record), and the rows of X, H and G go to shared memory
// as they are, 16 bytes at a time by cp.async. One stage holds a chunk's X, H1..H5, G0..G4, G5 (92
// feature groups, 94 KB); the next chunk's loads run during this chunk's MMAs. A layer with 64 inputs
// still reads 128 rows: rows past its inputs are the following groups' data, and the accumulator
// lanes that they give are never read. The six accumulators (336 TMEM columns) stay resident while
// the CTA walks its chunks.
// Bound by the loads (1.47 KB a record from L2): 65,536 records in 29 us; 39 us with H and G by records, 121 us
// when each record's features were scattered into K-major operands with 2-byte shared-memory stores.
constexpr uint32_t WG_TC_THREADS = 256, WG_TC_CHUNK = 64, WG_TC_TMEM = 512;
constexpr uint32_t WG_X = IN / 8, WG_H = ACT / 8, WG_G = GRAD / 8; // 16-byte groups of a record: 10, 40, 42
// a group's records, and 16 bytes that spread the groups of a record over the banks
constexpr uint32_t WG_GROUP = WG_TC_CHUNK * 16 + 16;
constexpr uint32_t WG_STAGE = (WG_X + WG_H + WG_G) * WG_GROUP, WG_TC_SMEM = 2 * WG_STAGE;
static_assert(WG_X + 8 * 4 + 16 <= WG_X + WG_H + WG_G, "the last layer's 128 operand rows stay in the stage");

__device__ __forceinline__ uint32_t tmem_col(int l) { return l < NLAYER - 1 ? 64u * (uint32_t)l : 320u; }

// groups [g0, g0 + GROUPS) of a stage: rows [r0, r0 + 64) of src (GROUPS x 16 bytes each, by records or by
// tiles as k_train_tc_wg stores them), zeros past n
template<uint32_t GROUPS, bool TILED>
__device__ __forceinline__ void wg_load(const uint32_t *__restrict__ src, uint32_t r0, uint32_t n, uint32_t dst)
{
    for(uint32_t i = threadIdx.x; i < GROUPS * WG_TC_CHUNK; i += WG_TC_THREADS)
    {
        const uint32_t s = TILED ? i % WG_TC_CHUNK : i / GROUPS, p = TILED ? i / WG_TC_CHUNK : i - s * GROUPS;
        const bool valid = r0 + s < n;
        const size_t group = TILED ? tiled_group(r0 + s, GROUPS, p) : (size_t)(r0 + s) * GROUPS + p;
        tc::cp_async16(dst + p * WG_GROUP + s * 16u, src + (valid ? group * 4u : 0u), valid);
    }
}

template<bool TILED> // H and G by tiles
__global__ void __launch_bounds__(WG_TC_THREADS)
        k_wgrad_tc(const uint32_t *__restrict__ X, const uint32_t *__restrict__ H, const uint32_t *__restrict__ G,
                   uint32_t n_cap, const uint32_t *__restrict__ d_n, float *__restrict__ dW, uint32_t *__restrict__ err)
{
    extern __shared__ __align__(1024) uint8_t smem[];
    __shared__ uint64_t mbar[2];
    __shared__ uint32_t tslot;
    const uint32_t tid = threadIdx.x, warp = tid >> 5, h = tid >> 7;
    const uint32_t n = d_n ? min(*d_n, n_cap) : n_cap;
    const uint32_t chunks = (n + WG_TC_CHUNK - 1) / WG_TC_CHUNK;
    const uint32_t base = tc::smem_addr(smem);
    auto load = [&](uint32_t c, uint32_t b) {
        const uint32_t r0 = c * WG_TC_CHUNK, st = base + b * WG_STAGE;
        wg_load<WG_X, false>(X, r0, n, st);
        wg_load<WG_H, TILED>(H, r0, n, st + WG_X * WG_GROUP);
        wg_load<WG_G, TILED>(G, r0, n, st + (WG_X + WG_H) * WG_GROUP);
    };
    if(blockIdx.x < chunks) load(blockIdx.x, 0);
    tc::cp_async_commit();
    if(warp == 0) tc::tmem_alloc(&tslot, WG_TC_TMEM);
    if(tid == 0)
    {
        tc::mbar_init(&mbar[0], 1);
        tc::mbar_init(&mbar[1], 1);
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tslot;
    uint32_t phase[2] = {0u, 0u}, k = 0;
    bool failed = false;
    for(uint32_t c = blockIdx.x; c < chunks; c += gridDim.x, ++k)
    {
        const uint32_t b = k & 1u, o = b ^ 1u;
        if(k > 0)
        {
            // the chunk before read the other stage: its MMAs must be done before that is refilled
            const bool ok = tc::mbar_wait(&mbar[o], phase[o]);
            if(__syncthreads_or(!ok))
            {
                failed = true;
                break;
            }
            phase[o] ^= 1u;
        }
        if(c + gridDim.x < chunks) load(c + gridDim.x, o);
        tc::cp_async_commit();
        tc::cp_async_wait<1>(); // this chunk's own groups have landed
        tc::fence_async_smem();
        tc::fence_before_sync();
        __syncthreads();
        if(tid == 0)
        {
            tc::fence_after_sync();
            const uint32_t st = base + b * WG_STAGE, gr = st + (WG_X + WG_H) * WG_GROUP;
            for(int l = 0; l < NLAYER; ++l)
            {
                const uint32_t idesc = tc::idesc_bf16(128, layer_out(l)) | tc::IDESC_A_MN | tc::IDESC_B_MN;
                const uint32_t a0 = l == 0 ? st : st + (WG_X + 8u * (l - 1)) * WG_GROUP, b0 = gr + 8u * l * WG_GROUP;
                for(uint32_t q = 0; q < WG_TC_CHUNK / 16; ++q)
                    tc::mma_bf16(tmem + tmem_col(l), tc::smem_desc(a0 + 256u * q, 128u, WG_GROUP),
                                 tc::smem_desc(b0 + 256u * q, 128u, WG_GROUP), idesc, k > 0 || q > 0);
            }
            tc::mma_commit(&mbar[b]);
        }
    }
    tc::cp_async_wait<0>();
    // the last chunk's MMAs (after a wait that ran out: the chunk's before it, once more)
    if(k > 0)
    {
        const uint32_t b = (k - 1u) & 1u;
        const bool ok = tc::mbar_wait(&mbar[b], phase[b]);
        if(__syncthreads_or(!ok)) failed = true;
    }
    if(failed)
    {
        if(tid == 0) atomicOr(err, TC_TIMEOUT);
    }
    else if(k > 0)
    {
        tc::fence_after_sync();
        // lane r = 32 (warp mod 4) + lane of TMEM holds row r of every layer's accumulator
        const uint32_t r = 32u * (warp & 3u) + (tid & 31u), lane_base = (32u * (warp & 3u)) << 16;
#pragma unroll 1
        for(int l = 0; l < NLAYER; ++l)
        {
            const uint32_t K = layer_in(l), N = layer_out(l);
            for(uint32_t c0 = 16u * h; c0 < N; c0 += 32u)
            {
                float v[16];
                tc::tmem_ld16(tmem + lane_base + tmem_col(l) + c0, v);
                tc::tmem_ld_wait();
                float4 *out = reinterpret_cast<float4 *>(dW + layer_off(l) + r * N + c0);
                if(r < K)
#pragma unroll
                    for(int j = 0; j < 4; ++j)
                        atomicAdd(out + j, make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]));
            }
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if(warp == 0) tc::tmem_dealloc(tmem, WG_TC_TMEM);
}

}// namespace

vkg_status nrc_wgrad_tc(vkg_ctx *ctx, const uint32_t *X, const uint32_t *H, const uint32_t *G, uint32_t n,
                        const uint32_t *d_n, bool tiled, float *dW, uint32_t *err, cudaStream_t st)
{
    if(n == 0) return VKG_OK;
    auto kern = tiled ? k_wgrad_tc<true> : k_wgrad_tc<false>;
    VKG_TRY_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)WG_TC_SMEM));
    const uint32_t chunks = (n + WG_TC_CHUNK - 1) / WG_TC_CHUNK;
    const uint32_t grid = std::min<uint32_t>(chunks, (uint32_t)ctx->num_sms);
    kern<<<grid, WG_TC_THREADS, WG_TC_SMEM, st>>>(X, H, G, n, d_n, dW, err);
    return cuda_check(ctx, cudaGetLastError(), "k_wgrad_tc");
}

// grid of a warpgroup kernel: a CTA per NWG tiles, at most as many as are resident
template<int NWG, class K>
vkg_status warpgroup_grid(vkg_ctx *ctx, K kern, uint32_t smem, uint32_t n, uint32_t &grid)
{
    VKG_TRY_CUDA(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 0;
    VKG_TRY_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, NWG * 128, smem));
    // TMEM: a resident CTA holds its share of the SM's 512 columns
    per_sm = std::max(1, std::min(per_sm, (int)(512 / tmem_columns(TC_WG_COLS, NWG))));
    const uint32_t tiles = (n + TC_TILE - 1) / TC_TILE;
    grid = std::min<uint32_t>((tiles + NWG - 1) / NWG, (uint32_t)(ctx->num_sms * per_sm));
    return VKG_OK;
}

template<int NWG>
vkg_status launch_forward_tc(vkg_ctx *ctx, const uint16_t *wtc, const uint32_t *X, uint32_t n, const uint32_t *d_n,
                             float *Y, uint32_t *err, cudaStream_t st)
{
    const uint32_t smem = TC_W_BYTES + NWG * TC_A_BYTES;
    uint32_t grid = 0;
    if(vkg_status s = warpgroup_grid<NWG>(ctx, k_infer_tc_wg<NWG>, smem, n, grid); s != VKG_OK) return s;
    k_infer_tc_wg<NWG><<<grid, NWG * 128, smem, st>>>(X, n, d_n, wtc, Y, err);
    return cuda_check(ctx, cudaGetLastError(), "k_infer_tc_wg");
}

// the pipelined MLP over encoded inputs X
static vkg_status nrc_forward_tc(vkg_ctx *ctx, const uint16_t *wtc, const uint32_t *X, uint32_t n, const uint32_t *d_n,
                                 float *Y, uint32_t *err, cudaStream_t st)
{
    // tiles in flight per SM (inference with the encoding, 4,096 / 20,000 / 65,536 / 2,073,600 queries: one
    // warpgroup a CTA 19 / 28 / 46 / 908 us, two 21 / 25 / 42 / 751, four 24 / 29 / 40 / 643, five 26 / 31 /
    // 42 / 684)
    const uint32_t tiles = (n + TC_TILE - 1) / TC_TILE, sms = (uint32_t)ctx->num_sms;
    if(tiles >= 3 * sms) return launch_forward_tc<4>(ctx, wtc, X, n, d_n, Y, err, st);
    if(tiles <= sms / 2) return launch_forward_tc<1>(ctx, wtc, X, n, d_n, Y, err, st);
    return launch_forward_tc<2>(ctx, wtc, X, n, d_n, Y, err, st);
}

template<int NWG>
vkg_status launch_train_tc(vkg_ctx *ctx, const uint16_t *wtc, const uint16_t *wtc_t, const uint32_t *X, const float *T,
                           uint32_t n, const uint32_t *d_n, uint32_t *H, uint32_t *G, float *dXg, float *loss,
                           uint32_t *err, cudaStream_t st)
{
    const uint32_t smem = 2 * TC_W_BYTES + NWG * (TC_A_BYTES + TC_G_BYTES);
    uint32_t grid = 0;
    if(vkg_status s = warpgroup_grid<NWG>(ctx, k_train_tc_wg<NWG>, smem, n, grid); s != VKG_OK) return s;
    k_train_tc_wg<NWG><<<grid, NWG * 128, smem, st>>>(X, T, n, d_n, wtc, wtc_t, reinterpret_cast<uint4 *>(H),
                                                      reinterpret_cast<uint4 *>(G), reinterpret_cast<float4 *>(dXg), loss,
                                                      err);
    return cuda_check(ctx, cudaGetLastError(), "k_train_tc_wg");
}

vkg_status nrc_train_tc(vkg_ctx *ctx, const uint16_t *wtc, const uint16_t *wtc_t, const uint32_t *X, const float *T,
                        uint32_t n, const uint32_t *d_n, uint32_t *H, uint32_t *G, float *dXg, float *loss,
                        uint32_t *err, cudaStream_t st)
{
    if(n == 0) return VKG_OK;
    const uint32_t tiles = (n + TC_TILE - 1) / TC_TILE, sms = (uint32_t)ctx->num_sms;
    // a wave that holds every tile, with as few tiles per SM as that takes (backward of 12,000 / 30,000 / 40,000 /
    // 65,536 records: one warpgroup a CTA 56 / 98 / 119 / 152 us, two 58 / 88 / 112 / 132, four 62 / 94 / 106 / 127)
    if(tiles > 2 * sms) return launch_train_tc<4>(ctx, wtc, wtc_t, X, T, n, d_n, H, G, dXg, loss, err, st);
    if(tiles > sms) return launch_train_tc<2>(ctx, wtc, wtc_t, X, T, n, d_n, H, G, dXg, loss, err, st);
    return launch_train_tc<1>(ctx, wtc, wtc_t, X, T, n, d_n, H, G, dXg, loss, err, st);
}

vkg_status nrc_infer_tc(vkg_ctx *ctx, const grid_config &gc, const __half2 *grid, const uint16_t *wtc,
                        const float *feats, const uint32_t *X, uint32_t n, const uint32_t *d_n, float *Y, uint32_t *err,
                        cudaStream_t st)
{
    if(n == 0) return VKG_OK;
    if(X) return nrc_forward_tc(ctx, wtc, X, n, d_n, Y, err, st);
    VKG_TRY_CUDA(ctx, cudaFuncSetAttribute(k_infer_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)TC_SMEM));
    int per_sm = 0;
    VKG_TRY_CUDA(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_infer_tc, TC_INFER_THREADS, TC_SMEM));
    // TMEM: every resident CTA holds 64 of the SM's 512 columns
    per_sm = std::max(1, std::min(per_sm, (int)(512 / TC_TMEM_COLS)));
    const uint32_t tiles = (n + TC_TILE - 1) / TC_TILE;
    const uint32_t grid_n = std::min<uint32_t>(tiles, (uint32_t)(ctx->num_sms * per_sm));
    k_infer_tc<<<grid_n, TC_INFER_THREADS, TC_SMEM, st>>>(feats, n, d_n, gc, grid, wtc, Y, err);
    return cuda_check(ctx, cudaGetLastError(), "k_infer_tc");
}

}// namespace nrc
}// namespace vkg

using namespace vkg;

extern "C" vkg_status vkg_diag_wait_timeout(vkg_ctx *ctx, uint32_t num_ctas, uint64_t limit_ns, uint32_t *d_err,
                                            uint64_t *d_elapsed_ns, void *stream)
{
    if(!ctx) return VKG_ERR_INVALID_ARGUMENT;
    if(!d_err || !d_elapsed_ns || num_ctas == 0 || num_ctas > 4096 || limit_ns == 0 || limit_ns > 100000000ull)
        return set_error(ctx, VKG_ERR_INVALID_ARGUMENT,
                         "vkg_diag_wait_timeout: need 1 <= num_ctas <= 4096 and 0 < limit_ns <= 1e8");
    if(vkg_status s = bind_device(ctx); s != VKG_OK) return s;
    nrc::k_wait_probe<<<num_ctas, nrc::TC_THREADS, 0, static_cast<cudaStream_t>(stream)>>>(
            limit_ns, d_err, reinterpret_cast<unsigned long long *>(d_elapsed_ns));
    return cuda_check(ctx, cudaGetLastError(), "k_wait_probe");
}

extern "C" vkg_status vkg_diag_tc_gemm(vkg_ctx *ctx, const uint16_t *d_a, const uint16_t *d_b, uint32_t k,
                                       uint32_t n, float *d_d, uint32_t *d_err, void *stream)
{
    if(!ctx) return VKG_ERR_INVALID_ARGUMENT;
    if(!d_a || !d_b || !d_d || !d_err || k == 0 || k % 16 || k > 256 || n < 16 || n > nrc::TC_TMEM_COLS || n % 16)
        return set_error(ctx, VKG_ERR_INVALID_ARGUMENT, "vkg_diag_tc_gemm: need 16 <= n <= 64, k <= 256, multiples of 16");
    if(vkg_status s = bind_device(ctx); s != VKG_OK) return s;
    const uint32_t smem = nrc::TC_TILE * k * 2 + n * k * 2;
    VKG_TRY_CUDA(ctx, cudaFuncSetAttribute(nrc::k_tc_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    nrc::k_tc_gemm<<<1, nrc::TC_THREADS, smem, static_cast<cudaStream_t>(stream)>>>(d_a, d_b, k, n, d_d, d_err);
    return cuda_check(ctx, cudaGetLastError(), "k_tc_gemm");
}
