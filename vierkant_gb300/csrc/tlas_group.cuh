// Eight lanes per ray through both levels (trace_tlas with the group traversal of traverse_group.cuh).
//
// A step tests eight boxes side by side: the children of a node of either level, or the world boxes of
// the instances of a top-level leaf, which is pushed as one entry and opened when it is popped. What the
// ray hits is ranked by entry distance and pushed, the nearest on top; a popped instance moves the ray to
// object space and goes on with its root, as tl_step does, above a RETURN marker. Hits and ties are those
// of trace_tlas: the nearest triangle, then the smaller instance, then the smaller triangle index.
//
// Two-level rays differ in length far more than single-level ones (8 of 32 lanes are active with one
// thread per ray) and the longest of them set the time; with four rays to a warp and a step split over
// eight lanes both shrink.
#pragma once

#include "tlas.cuh"
#include "traverse_group.cuh"

namespace vkg
{

// Largest batch traced by groups: 131,072 camera rays take 43 / 278 / 365 / 417 us by groups and 73 / 328 / 413 / 464
// a thread each over 50 / 4,000 / 20,000 / 40,000 instances of a flat scene (32,768 rays 29 / 108 / 139 / 167 and
// 60 / 240 / 341 / 342); 260,000 rays gain from a thread each.
// Closest-hit rays through instances that overlap a lot gain from it earlier, as groups leave them more lanes idle.
// The time of a thread each over that of groups, for 98,304 / 65,536 / 49,152 random rays: 0.6 / 0.8 / 1.0 where a
// line crosses 250 instance boxes on average (camera rays 1.0 / 1.2 / 1.4), 0.8 / 1.1 / 1.3 where it crosses 20 to
// 40 (camera rays 1.2 / 1.5 / 1.7); any-hit rays 0.9 or more at 98,304, 1.1 or more below.
constexpr uint32_t TL_GROUP_MAX_RAYS = 1u << 17, TL_GROUP_MAX_OVERLAPPING = 3u << 14;
constexpr float TL_GROUP_OVERLAP = 64.f;
inline uint32_t tl_group_max_rays(const vkg_tlas *t, bool any)
{
    return any || t->overlap <= TL_GROUP_OVERLAP ? TL_GROUP_MAX_RAYS : TL_GROUP_MAX_OVERLAPPING;
}

// Stack entries of a group. Every level leaves at most 7 entries behind and the last one 8; between the
// levels an opened leaf adds 8 and the marker 1: 7 (top depth + mesh depth) + 4. The shared memory of
// the deepest trees the builds allow costs shallow ones 2-4 %.
constexpr int TL_GROUP_SMALL_STACK = 96, TL_GROUP_STACK = 208;
static_assert(7 * (TLAS_MAX_DEPTH + (TRAVERSAL_STACK - 1) / 7 + 1) + 4 <= (uint32_t)TL_GROUP_STACK, "deepest trees fit");
inline bool tl_group_small_stack(const vkg_tlas *t)
{
    return 7 * (t->top.depth + t->max_blas_depth) + 4 <= (uint32_t)TL_GROUP_SMALL_STACK;
}

// All 32 lanes of a warp call this together; `active`, the ray and `st` are uniform over a group. STACK:
// entries of `st`.
template<bool ANY, int STACK>
__device__ __forceinline__ tlas_result trace_tlas_group(bool active, const node8 *__restrict__ tnodes,
                                                        const inst_rec *__restrict__ inst,
                                                        const float4 *__restrict__ box,
                                                        const blas_ref *__restrict__ blas, float ox, float oy, float oz,
                                                        float tmin, float dx, float dy, float dz, float tmax, int cull,
                                                        uint2 *st)
{
    constexpr uint32_t ALL = 0xffffffffu, GROUP = 0xFFu;
    const uint32_t lane = threadIdx.x & 31u, k = lane & 7u, g0 = lane & 24u;
    float o[3] = {ox, oy, oz}, d[3] = {dx, dy, dz}, inv[3];
    const float winv[3] = {safe_rcp(dx), safe_rcp(dy), safe_rcp(dz)};
    for(int a = 0; a < 3; ++a) inv[a] = winv[a];
    float best_t = tmax, mu = 0.f, mv = 0.f;
    uint32_t best = VKG_MISS, best_inst = VKG_MISS, cur_inst = VKG_MISS;
    const node8 *nodes = tnodes;
    const tri_rec *tris = nullptr;
    bool in_blas = false, mine = false, occluded = false;
    int sp = active ? 1 : 0;
    if(active && k == 0) st[0] = make_uint2(0u, __float_as_uint(tmin));
    __syncwarp();
    for(;;)
    {
        uint32_t ni = 0;    // the node, or the first instance of an opened leaf
        uint32_t boxes = 0; // instances of an opened leaf (at most 8); 0: a node
        // what goes back on the stack in the place of the popped entry. Lane 0 writes it after the vote below:
        // until then the group's other lanes may still have to read that place
        uint2 back = make_uint2(0u, 0u);
        bool have = false, put = false;
        while(sp > 0 && !have)
        {
            const uint2 e = st[--sp];
            if(e.x == TL_RETURN)
            {
                o[0] = ox, o[1] = oy, o[2] = oz;
                d[0] = dx, d[1] = dy, d[2] = dz;
                for(int a = 0; a < 3; ++a) inv[a] = winv[a];
                nodes = tnodes;
                in_blas = false;
                continue;
            }
            if(__uint_as_float(e.y) > best_t) continue;
            ni = e.x;
            if(!(e.x & LEAF_BIT))
            {
                have = true;
                continue;
            }
            // (leaves on the stack are the top level's)
            ni = e.x & 0x07FFFFFFu;
            const uint32_t cnt = ((e.x >> 27) & 0xFu) + 1u;
            if(cnt > 1)
            {
                boxes = min(cnt, (uint32_t)GROUP_LANES);
                if(cnt > GROUP_LANES) // the rest of a large leaf waits below
                {
                    back = make_uint2(LEAF_BIT | ((cnt - GROUP_LANES - 1u) << 27) | (ni + GROUP_LANES), e.y);
                    put = true;
                }
                have = true;
                continue;
            }
            const float4 *mp = reinterpret_cast<const float4 *>(inst + ni);
            const uint4 meta = __ldg(reinterpret_cast<const uint4 *>(mp + 6));
            const blas_ref B = blas[meta.x];
            if(B.num_tris == 0 || sp + 1 >= STACK) continue;
            const float4 m[3] = {__ldg(mp), __ldg(mp + 1), __ldg(mp + 2)};
            to_object(m, ox, oy, oz, dx, dy, dz, o, d);
            for(int a = 0; a < 3; ++a) inv[a] = safe_rcp(d[a]);
            nodes = B.nodes;
            tris = B.tris;
            cur_inst = meta.y;
            in_blas = true;
            back = make_uint2(TL_RETURN, __float_as_uint(tmin));
            put = true;
            ni = 0;
            have = true;
        }
        if(!__any_sync(ALL, have)) break;
        if(put && k == 0) st[sp] = back;
        sp += put ? 1 : 0; // (a branch around both lines, or a barrier of the group in the loop, cost 0.7-1.3 % more)
        float tn, tf;
        uint32_t word;
        bool hit;
        if(boxes)
        {
            const uint32_t i = ni + min(k, boxes - 1u);
            const float4 b0 = __ldg(box + 2 * (size_t)i), b1 = __ldg(box + 2 * (size_t)i + 1);
            const float x0 = (b0.x - o[0]) * inv[0], x1 = (b0.w - o[0]) * inv[0];
            const float y0 = (b0.y - o[1]) * inv[1], y1 = (b1.x - o[1]) * inv[1];
            const float z0 = (b0.z - o[2]) * inv[2], z1 = (b1.y - o[2]) * inv[2];
            tn = fmaxf(fmaxf(fminf(x0, x1), fminf(y0, y1)), fmaxf(fminf(z0, z1), tmin));
            tf = fminf(fminf(fmaxf(x0, x1), fmaxf(y0, y1)), fminf(fmaxf(z0, z1), best_t));
            word = LEAF_BIT | i;
            hit = k < boxes && tn <= tf;
        }
        else
        {
            const uint8_t *np = reinterpret_cast<const uint8_t *>(nodes + ni);
            const uint4 w0 = __ldg(reinterpret_cast<const uint4 *>(np));
            word = __ldg(reinterpret_cast<const uint32_t *>(np + 64) + k);
            float near[3], far[3];
#pragma unroll
            for(int a = 0; a < 3; ++a)
            {
                const uint32_t lo = 16u + 8u * a + k, hi = lo + 24u;
                const float q0 = (float)__ldg(np + (inv[a] < 0.f ? hi : lo)), q1 = (float)__ldg(np + (inv[a] < 0.f ? lo : hi));
                const float org = __uint_as_float(a == 0 ? w0.x : a == 1 ? w0.y : w0.z);
                const float to = __fmul_rn(__fsub_rn(org, o[a]), inv[a]);
                const float s = __fmul_rn(exp_scale((w0.w >> (8 * a)) & 0xFFu), inv[a]);
                near[a] = fmaf(q0, s, to);
                far[a] = fmaf(q1, s, to);
            }
            tn = fmaxf(fmaxf(near[0], near[1]), fmaxf(near[2], tmin));
            tf = fminf(fminf(far[0], far[1]), fminf(far[2], best_t));
            hit = have && k < (w0.w >> 24) && tn <= tf;
        }
        const bool leaf = hit && in_blas && (word & LEAF_BIT), push = hit && !leaf;
        const uint32_t key = child_key<false>(tn, k), rank = push ? key : 0u;
        int farther = 0;
#pragma unroll
        for(int q = 1; q < GROUP_LANES; ++q) farther += __shfl_xor_sync(ALL, rank, q) > key ? 1 : 0;
        const int pushed = __popc((__ballot_sync(ALL, push) >> g0) & GROUP);
        if(push && sp + farther < STACK)
            st[sp + farther] = make_uint2(word, __float_as_uint(key_dist<false>(key)));
        sp = min(sp + pushed, STACK);
        if(__any_sync(ALL, leaf))
        {
            float ct = best_t, cu = 0.f, cv = 0.f;
            uint32_t cp = best, ci = best_inst;
            bool better = false;
            const uint32_t cnt = leaf ? ((word >> 27) & 0xFu) + 1u : 0u;
            const float4 *tp = reinterpret_cast<const float4 *>(tris + (word & 0x07FFFFFFu));
            for(uint32_t i = 0; i < cnt && !(ANY && better); ++i, tp += 3)
            {
                const float4 a = __ldg(tp), b = __ldg(tp + 1), c = __ldg(tp + 2);
                const int tcull = cull == CULL_BACK ||
                                  (cull == CULL_BACK_UNLESS_TWOSIDED && !(__float_as_uint(c.z) & TRI_FLAG_TWOSIDED));
                float t, u, v;
                if(!tri_test(a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, c.x, o[0], o[1], o[2], d[0], d[1], d[2], tcull, t, u,
                             v))
                    continue;
                if(!(t > tmin && t < tmax)) continue;
                const uint32_t prim = __float_as_uint(c.y);
                if(!ANY && !(t < ct || (t == ct && (cur_inst < ci || (cur_inst == ci && prim < cp))))) continue;
                better = true;
                ct = t;
                cp = prim;
                ci = cur_inst;
                cu = u;
                cv = v;
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
                uint32_t gp = cp, gi = ci;
#pragma unroll
                for(int q = 1; q < GROUP_LANES; q <<= 1)
                {
                    const float t2 = __shfl_xor_sync(ALL, gt, q);
                    const uint32_t p2 = __shfl_xor_sync(ALL, gp, q), i2 = __shfl_xor_sync(ALL, gi, q);
                    if(t2 < gt || (t2 == gt && (i2 < gi || (i2 == gi && p2 < gp))))
                    {
                        gt = t2;
                        gp = p2;
                        gi = i2;
                    }
                }
                if(gp != best || gi != best_inst || gt != best_t)
                {
                    mine = better && cp == gp && ci == gi && ct == gt;
                    if(mine)
                    {
                        mu = cu;
                        mv = cv;
                    }
                }
                best = gp;
                best_inst = gi;
                best_t = gt;
            }
        }
        __syncwarp(); // the pushed entries are visible to the group
    }
    tlas_result r;
    r.occluded = occluded;
    r.prim = best;
    r.inst = best_inst;
    const uint32_t own = (__ballot_sync(ALL, mine) >> g0) & GROUP, src = g0 + (own ? __ffs(own) - 1u : 0u);
    const float u = __shfl_sync(ALL, mu, src), v = __shfl_sync(ALL, mv, src);
    r.t = best == VKG_MISS ? 0.f : best_t;
    r.u = best == VKG_MISS ? 0.f : u;
    r.v = best == VKG_MISS ? 0.f : v;
    return r;
}

}// namespace vkg
