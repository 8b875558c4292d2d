// Eight lanes per ray: the traversal of traverse.cuh for batches too small to fill the GPU with one
// thread per ray.
//
// There a ray's own chain of dependent steps sets the time: per node a line from L2, 300 instructions
// for eight children, and the triangles of its leaves one after the other; and a warp takes as many
// steps as the longest of its 32 rays. Here lane k of a ray's eight tests child k and, where that is a leaf
// the ray hits, its triangles: a node costs two L2 latencies and a third of the instructions, and a
// warp waits for the longest of four rays. The group's stack is in shared memory; children are ranked
// with shuffles and pushed side by side. (Four lanes of two children each measured 31 against 24 us for
// 1,000 rays and 112 against 120 us for 100,000: not worth a second variant. Prefetching the pushed
// children's nodes into L1 cost 3-20 %.)
//
// The nodes a ray visits and the hit it reports are those of ray_step(): the same slab tests, keys and
// stack order; of a node's leaves all triangles are tested instead of stopping at the first leaf that
// starts behind the best hit, which cannot hold a nearer one.
#pragma once

#include "traverse.cuh"

namespace vkg
{

// a group's stack; the pad entry spreads the groups of a warp over the banks
template<int STACK>
constexpr int group_stack_entries = STACK + 1;
constexpr int GROUP_LANES = 8;
// Largest batch traced by groups, below the first scenes' break-even: over seven scenes (Cornell boxes, an icosphere, a
// terrain, loose triangles) 16,384 rays are 1.8-3.1 times as fast as with a thread each, 65,536 random rays 1.1-1.5
// and camera rays 1.6-2.1 times, 81,920 random rays 0.93-1.4 times, 150,000 take 128-171 against 115-130 us.
constexpr uint32_t GROUP_MAX_RAYS = 1u << 16;

// All 32 lanes of a warp call this together; `active`, the ray and `st` are uniform over a group's
// lanes. The result is uniform over the group.
// f: the candidate filter (no_filter, traverse.cuh); what it accepts does not depend on the order of the tests.
template<bool ANY, int STACK, class F = no_filter>
__device__ __forceinline__ trace_result trace_group(bool active, const node8 *__restrict__ nodes,
                                                    const tri_rec *__restrict__ tris, float ox, float oy, float oz,
                                                    float tmin, float dx, float dy, float dz, float tmax, int cull,
                                                    uint2 *st, unsigned long long *__restrict__ counters,
                                                    const F &f = F())
{
    constexpr uint32_t ALL = 0xffffffffu, GROUP = 0xFFu;
    const uint32_t lane = threadIdx.x & 31u, k = lane & 7u, g0 = lane & 24u;
    const float ix = safe_rcp(dx), iy = safe_rcp(dy), iz = safe_rcp(dz);
    // byte offsets of this lane's child in the near and far planes' quantised coordinates
    const uint32_t nx = (ix < 0.f ? 40u : 16u) + k, ny = (iy < 0.f ? 48u : 24u) + k, nz = (iz < 0.f ? 56u : 32u) + k;
    const uint32_t fx = 56u + 2u * k - nx, fy = 72u + 2u * k - ny, fz = 88u + 2u * k - nz;
    float best_t = tmax, mu = 0.f, mv = 0.f;
    uint32_t best = VKG_MISS;
    bool mine = false, occluded = false; // mine: this lane holds the best hit's barycentric coordinates
    int sp = active ? 1 : 0;
    if(active && k == 0) st[0] = make_uint2(0u, __float_as_uint(tmin));
    __syncwarp();
    for(;;)
    {
        uint32_t ni = 0;
        bool have = false;
        while(sp > 0 && !have)
        {
            const uint2 e = st[--sp];
            ni = e.x;
            have = !(__uint_as_float(e.y) > best_t);
        }
        if(!__any_sync(ALL, have)) break;
        const uint8_t *np = reinterpret_cast<const uint8_t *>(nodes + (have ? ni : 0u));
        const uint4 w0 = __ldg(reinterpret_cast<const uint4 *>(np));
        const uint32_t child = __ldg(reinterpret_cast<const uint32_t *>(np + 64) + k);
        const float qnx = (float)__ldg(np + nx), qny = (float)__ldg(np + ny), qnz = (float)__ldg(np + nz);
        const float qfx = (float)__ldg(np + fx), qfy = (float)__ldg(np + fy), qfz = (float)__ldg(np + fz);
        const float tox = __fmul_rn(__fsub_rn(__uint_as_float(w0.x), ox), ix);
        const float toy = __fmul_rn(__fsub_rn(__uint_as_float(w0.y), oy), iy);
        const float toz = __fmul_rn(__fsub_rn(__uint_as_float(w0.z), oz), iz);
        const float sx = __fmul_rn(exp_scale(w0.w & 0xFFu), ix), sy = __fmul_rn(exp_scale((w0.w >> 8) & 0xFFu), iy),
                    sz = __fmul_rn(exp_scale((w0.w >> 16) & 0xFFu), iz);
        const float tn = fmaxf(fmaxf(fmaf(qnx, sx, tox), fmaf(qny, sy, toy)), fmaxf(fmaf(qnz, sz, toz), tmin));
        const float tf = fminf(fminf(fmaf(qfx, sx, tox), fmaf(qfy, sy, toy)), fminf(fmaf(qfz, sz, toz), best_t));
        const bool hit = have && k < (w0.w >> 24) && tn <= tf;
        const bool inner = hit && !(child & LEAF_BIT), leaf = hit && (child & LEAF_BIT);
        // internal children: the nearest on top of the stack (no ordered key is 0)
        const uint32_t key = child_key<false>(tn, k), rank = inner ? key : 0u;
        int farther = 0;
#pragma unroll
        for(int o = 1; o < GROUP_LANES; ++o) farther += __shfl_xor_sync(ALL, rank, o) > key ? 1 : 0;
        const int pushed = __popc((__ballot_sync(ALL, inner) >> g0) & GROUP);
        if(inner)
        {
            const int pos = sp + farther;
            if(pos < STACK) st[pos] = make_uint2(child, __float_as_uint(key_dist<false>(key)));
            else if(counters) atomicOr(&counters[2], 1ull);
        }
        sp = min(sp + pushed, STACK);
        if(__any_sync(ALL, leaf))
        {
            float ct = best_t, cu = 0.f, cv = 0.f;
            uint32_t cp = best;
            bool better = false;
            const uint32_t cnt = leaf ? ((child >> 27) & 0xFu) + 1u : 0u;
            const float4 *tp = reinterpret_cast<const float4 *>(tris + (child & 0x07FFFFFFu));
            auto test = [&](const float4 &a, const float4 &b, const float4 &c) {
                const int tcull = cull == CULL_BACK ||
                                  (cull == CULL_BACK_UNLESS_TWOSIDED && !(__float_as_uint(c.z) & TRI_FLAG_TWOSIDED));
                float t, u, v;
                if(!tri_test(a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, c.x, ox, oy, oz, dx, dy, dz, tcull, t, u, v))
                    return;
                if(!(t > tmin && t < tmax)) return;
                const uint32_t prim = __float_as_uint(c.y);
                if(!ANY && !(t < ct || (t == ct && prim < cp))) return;
                if(F::active && (__float_as_uint(c.z) & TRI_FLAG_ALPHA) && !f.accept(0u, prim, u, v)) return;
                better = true;
                ct = t;
                cp = prim;
                cu = u;
                cv = v;
            };
            // two triangles' records in flight
            for(uint32_t i = 0; i < cnt && !(ANY && better); i += 2, tp += 6)
            {
                const float4 a0 = __ldg(tp), b0 = __ldg(tp + 1), c0 = __ldg(tp + 2);
                float4 a1 = a0, b1 = b0, c1 = c0;
                if(i + 1 < cnt)
                {
                    a1 = __ldg(tp + 3);
                    b1 = __ldg(tp + 4);
                    c1 = __ldg(tp + 5);
                }
                test(a0, b0, c0);
                if(i + 1 < cnt) test(a1, b1, c1);
            }
            const uint32_t won = __ballot_sync(ALL, better);
            if(ANY)
            {
                if((won >> g0) & GROUP)
                {
                    occluded = true;
                    sp = 0;
                }
            }
            else if(won)
            {
                float gt = ct;
                uint32_t gp = cp;
#pragma unroll
                for(int o = 1; o < GROUP_LANES; o <<= 1)
                {
                    const float t2 = __shfl_xor_sync(ALL, gt, o);
                    const uint32_t p2 = __shfl_xor_sync(ALL, gp, o);
                    if(t2 < gt || (t2 == gt && p2 < gp))
                    {
                        gt = t2;
                        gp = p2;
                    }
                }
                // (a triangle sits in one leaf: one lane of the group has the new best)
                if(gp != best || gt != best_t)
                {
                    mine = better && cp == gp && ct == gt;
                    if(mine)
                    {
                        mu = cu;
                        mv = cv;
                    }
                }
                best = gp;
                best_t = gt;
            }
        }
        __syncwarp(); // the pushed entries are visible to the group
    }
    trace_result r;
    r.occluded = occluded;
    r.prim = best;
    const uint32_t own = (__ballot_sync(ALL, mine) >> g0) & GROUP, src = g0 + (own ? __ffs(own) - 1u : 0u);
    const float u = __shfl_sync(ALL, mu, src), v = __shfl_sync(ALL, mv, src);
    r.t = best == VKG_MISS ? 0.f : best_t;
    r.u = best == VKG_MISS ? 0.f : u;
    r.v = best == VKG_MISS ? 0.f : v;
    return r;
}

}// namespace vkg
