// Stable LSD radix sort of (key, value) pairs, 8 bits per pass: per-tile digit histograms, an exclusive
// scan of every digit's counts over the tiles (one CTA per digit), and a scatter that adds the digits'
// first positions; ranks within a warp come from __match_any_sync. Used by the BVH builds (Morton
// codes).
//
// Bound by latency at the sizes of a scene's builds: a tile's steps follow one another, so sorts of up to
// SORT_SMALL keys take tiles of 4 keys a thread (20,000 keys: 5 tiles of 16 a thread took 21 us a
// scatter), larger ones 16, whose longer runs per digit write fewer partial lines. One CTA scanned all
// (digit, tile) counts before, 31 us a pass for 522,242 keys.
#pragma once

#include "internal.hpp"

namespace vkg
{
namespace
{

constexpr int SORT_THREADS = 256;
constexpr uint32_t SORT_SMALL = 1u << 20;
// keys per tile, and tiles, of a sort of n keys
__host__ __device__ constexpr uint32_t sort_items(uint32_t n) { return n <= SORT_SMALL ? 4u : 16u; }
__host__ __device__ constexpr uint32_t sort_tiles(uint32_t n)
{
    return (n + SORT_THREADS * sort_items(n) - 1) / (SORT_THREADS * sort_items(n));
}
// words of the count array: 256 rows of one count per tile, then the 256 digits' totals
__host__ __device__ constexpr size_t sort_count_words(uint32_t n) { return 256 * (size_t)sort_tiles(n) + 256; }

template<int ITEMS>
__global__ void __launch_bounds__(SORT_THREADS)
        k_radix_hist(const uint32_t *__restrict__ keys, uint32_t n, int shift, uint32_t *__restrict__ counts, uint32_t tiles)
{
    __shared__ uint32_t hist[256];
    hist[threadIdx.x] = 0;
    __syncthreads();
    const size_t base = (size_t)blockIdx.x * (SORT_THREADS * ITEMS);
    uint32_t key[ITEMS];
#pragma unroll
    for(int it = 0; it < ITEMS; ++it)
    {
        const size_t i = base + (size_t)it * SORT_THREADS + threadIdx.x;
        key[it] = i < n ? keys[i] : 0u;
    }
#pragma unroll
    for(int it = 0; it < ITEMS; ++it)
        if(base + (size_t)it * SORT_THREADS + threadIdx.x < n) atomicAdd(&hist[(key[it] >> shift) & 0xFFu], 1u);
    __syncthreads();
    counts[(size_t)threadIdx.x * tiles + blockIdx.x] = hist[threadIdx.x];
}

// inclusive scan over the block's 256 threads
__device__ __forceinline__ uint32_t scan256(uint32_t x, uint32_t (&warp_sums)[8])
{
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    for(int o = 1; o < 32; o <<= 1)
    {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if(lane >= (uint32_t)o) x += y;
    }
    if(lane == 31) warp_sums[warp] = x;
    __syncthreads();
    for(uint32_t w = 0; w < warp; ++w) x += warp_sums[w];
    __syncthreads();
    return x;
}

// CTA = digit: its row of counts becomes the exclusive scan over the tiles; totals[digit] = the sum
__global__ void __launch_bounds__(256) k_radix_scan(uint32_t *__restrict__ counts, uint32_t tiles)
{
    __shared__ uint32_t warp_sums[8];
    __shared__ uint32_t s_last;
    uint32_t *row = counts + (size_t)blockIdx.x * tiles, carry = 0;
    for(uint32_t base = 0; base < tiles; base += 256)
    {
        const uint32_t i = base + threadIdx.x, v = i < tiles ? row[i] : 0u;
        const uint32_t x = scan256(v, warp_sums);
        if(i < tiles) row[i] = carry + x - v;
        if(threadIdx.x == 255) s_last = x;
        __syncthreads();
        carry += s_last;
        __syncthreads();
    }
    if(threadIdx.x == 0) counts[256 * (size_t)tiles + blockIdx.x] = carry;
}

template<int ITEMS>
__global__ void __launch_bounds__(SORT_THREADS)
        k_radix_scatter(const uint32_t *__restrict__ keys_in, const uint32_t *__restrict__ vals_in, uint32_t n, int shift,
                        const uint32_t *__restrict__ counts, uint32_t tiles, uint32_t *__restrict__ keys_out,
                        uint32_t *__restrict__ vals_out)
{
    __shared__ uint32_t s_off[256];
    __shared__ uint32_t s_warp[8][257];
    __shared__ uint32_t warp_sums[8];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    // this tile's first position of every digit: the smaller digits' totals, then the tiles before
    const uint32_t total = counts[256 * (size_t)tiles + tid], before = counts[(size_t)tid * tiles + blockIdx.x];
    s_off[tid] = scan256(total, warp_sums) - total + before;
    const uint32_t lt_mask = (1u << lane) - 1u;
    const size_t base = (size_t)blockIdx.x * (SORT_THREADS * ITEMS);
    uint32_t key[ITEMS], val[ITEMS];
#pragma unroll
    for(int it = 0; it < ITEMS; ++it)
    {
        const size_t i = base + (size_t)it * SORT_THREADS + tid;
        key[it] = i < n ? keys_in[i] : 0u;
        val[it] = i < n ? vals_in[i] : 0u;
    }
#pragma unroll
    for(int it = 0; it < ITEMS; ++it)
    {
        for(uint32_t j = tid; j < 8u * 257u; j += SORT_THREADS) (&s_warp[0][0])[j] = 0u;
        __syncthreads();
        const bool valid = base + (size_t)it * SORT_THREADS + tid < n;
        const uint32_t digit = valid ? ((key[it] >> shift) & 0xFFu) : 256u;
        const uint32_t peers = __match_any_sync(0xffffffffu, digit);
        const uint32_t rank = __popc(peers & lt_mask);
        if(rank == 0) s_warp[warp][digit] = __popc(peers);
        __syncthreads();
        // exclusive prefix over the 8 warps for digit `tid`
        uint32_t run = 0;
        for(int w = 0; w < 8; ++w)
        {
            const uint32_t c = s_warp[w][tid];
            s_warp[w][tid] = run;
            run += c;
        }
        __syncthreads();
        if(valid)
        {
            const uint32_t pos = s_off[digit] + s_warp[warp][digit] + rank;
            keys_out[pos] = key[it];
            vals_out[pos] = val[it];
        }
        __syncthreads();
        s_off[tid] += run;
        __syncthreads();
    }
}

// the pairs (kin, vin) sorted by the low `bits` of their keys; the sorted arrays are in kin / vin, whose
// pointers change places with kout / vout as the passes go. counts: sort_count_words(n) words
inline void radix_sort(uint32_t *&kin, uint32_t *&vin, uint32_t *&kout, uint32_t *&vout, uint32_t n, int bits,
                       uint32_t *counts, cudaStream_t st)
{
    const uint32_t tiles = sort_tiles(n);
    for(int shift = 0; shift < bits; shift += 8)
    {
        if(sort_items(n) == 4) k_radix_hist<4><<<tiles, SORT_THREADS, 0, st>>>(kin, n, shift, counts, tiles);
        else k_radix_hist<16><<<tiles, SORT_THREADS, 0, st>>>(kin, n, shift, counts, tiles);
        k_radix_scan<<<256, 256, 0, st>>>(counts, tiles);
        if(sort_items(n) == 4)
            k_radix_scatter<4><<<tiles, SORT_THREADS, 0, st>>>(kin, vin, n, shift, counts, tiles, kout, vout);
        else
            k_radix_scatter<16><<<tiles, SORT_THREADS, 0, st>>>(kin, vin, n, shift, counts, tiles, kout, vout);
        uint32_t *k = kin, *v = vin;
        kin = kout;
        vin = vout;
        kout = k;
        vout = v;
    }
}

// ---- Karras radix tree ------------------------------------------------------------------------
__device__ __forceinline__ int kdelta(const uint32_t *codes, int64_t n, int64_t i, int64_t j)
{
    if(j < 0 || j >= n) return -1;
    uint32_t a = codes[i], b = codes[j];
    if(a == b) return 32 + __clz((uint32_t)i ^ (uint32_t)j);
    return __clz(a ^ b);
}


}// namespace
}// namespace vkg
