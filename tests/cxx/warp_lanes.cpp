// The traversals by groups of eight lanes (csrc/tlas_group.cuh, csrc/traverse_group.cuh), compiled for the host and
// run by 32 emulated lanes. The lanes of a warp meet only in the warp-wide operations: between two of them they may
// run in any order. Here every lane runs alone up to the next one, in the order of a permutation of
// the lanes, and the results have to be those of trace_tlas and trace_ray, one thread per ray, for every order.
#include <ucontext.h>

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <random>
#include <vector>

// ---- the lanes ----------------------------------------------------------------------------------
static constexpr int LANES = 32;
static ucontext_t g_main, g_lane[LANES];
static std::vector<char> g_stack[LANES];
static uint32_t g_arg[2][LANES]; // arguments of the operation under way and of the one before
static uint32_t g_ops[LANES];    // warp-wide operations a lane has entered
static int g_current;
static bool g_done[LANES];
static std::function<void(int)> g_body;
static struct
{
    unsigned x;
} threadIdx;

// every lane enters; returns once all have
static const uint32_t *meet(uint32_t value)
{
    const int me = g_current;
    uint32_t *const slot = g_arg[g_ops[me]++ & 1u];
    slot[me] = value;
    swapcontext(&g_lane[me], &g_main);
    return slot;
}
static void lane_main()
{
    g_body(g_current);
    g_done[g_current] = true;
}
static void run_warp(const int (&order)[LANES], const std::function<void(int)> &body)
{
    g_body = body;
    for(int l = 0; l < LANES; ++l)
    {
        g_stack[l].resize(1u << 18);
        getcontext(&g_lane[l]);
        g_lane[l].uc_stack.ss_sp = g_stack[l].data();
        g_lane[l].uc_stack.ss_size = g_stack[l].size();
        g_lane[l].uc_link = &g_main;
        makecontext(&g_lane[l], lane_main, 0);
        g_done[l] = false;
        g_ops[l] = 0;
    }
    for(bool left = true; left;)
    {
        left = false;
        for(int l: order)
            if(!g_done[l])
            {
                g_current = l;
                threadIdx.x = (unsigned)l;
                swapcontext(&g_main, &g_lane[l]);
                left = left || !g_done[l];
            }
        // a lane that is done while others still meet, or one that met more often: not one warp's program
        for(int l = 1; l < LANES; ++l)
            if(g_ops[l] != g_ops[0] || g_done[l] != g_done[0] || g_ops[0] > 100000u)
            {
                std::puts("the lanes left the common sequence of warp-wide operations, or do not come to an end");
                std::exit(1);
            }
    }
}

// ---- what the headers use of the device ---------------------------------------------------------
static inline uint32_t __float_as_uint(float f)
{
    uint32_t u;
    std::memcpy(&u, &f, 4);
    return u;
}
static inline float __uint_as_float(uint32_t u)
{
    float f;
    std::memcpy(&f, &u, 4);
    return f;
}
template<class T>
static inline T __ldg(const T *p)
{
    return *p;
}
static inline float __fmul_rn(float a, float b) { return a * b; }
static inline float __fsub_rn(float a, float b) { return a - b; }
static inline float __frcp_rn(float a) { return 1.f / a; }
static inline int __popc(uint32_t v) { return __builtin_popcount(v); }
static inline int __ffs(uint32_t v) { return __builtin_ffs((int)v); }
static inline uint32_t min(uint32_t a, uint32_t b) { return a < b ? a : b; }
static inline int min(int a, int b) { return a < b ? a : b; }
static inline uint32_t max(uint32_t a, uint32_t b) { return a > b ? a : b; }
static inline unsigned long long atomicOr(unsigned long long *p, unsigned long long v) { return *p |= v, 0ull; }
static inline uint32_t __ballot_sync(uint32_t, bool p)
{
    const uint32_t *a = meet(p);
    uint32_t m = 0;
    for(int l = 0; l < LANES; ++l) m |= a[l] << l;
    return m;
}
static inline bool __any_sync(uint32_t m, bool p) { return __ballot_sync(m, p) != 0u; }
static inline void __syncwarp(uint32_t = ~0u) { meet(0u); }
static inline uint32_t __shfl_sync(uint32_t, uint32_t v, uint32_t src) { return meet(v)[src & 31u]; }
static inline float __shfl_sync(uint32_t m, float v, uint32_t src)
{
    return __uint_as_float(__shfl_sync(m, __float_as_uint(v), src));
}
static inline uint32_t __shfl_xor_sync(uint32_t, uint32_t v, int o)
{
    const int me = g_current;
    return meet(v)[me ^ o];
}
static inline float __shfl_xor_sync(uint32_t m, float v, int o)
{
    return __uint_as_float(__shfl_xor_sync(m, __float_as_uint(v), o));
}

#include "../../vierkant_gb300/csrc/tlas_group.cuh"

using namespace vkg;

// ---- a small two-level scene ---------------------------------------------------------------------
struct box
{
    float lo[3], hi[3];
};
struct child
{
    box b;
    uint32_t word;
};

static node8 make_node(const std::vector<child> &c)
{
    node8 n;
    std::memset(&n, 0, sizeof(n));
    n.nchild = (uint8_t)c.size();
    for(int a = 0; a < 3; ++a)
    {
        float lo = c[0].b.lo[a], hi = c[0].b.hi[a];
        for(const child &k: c)
        {
            lo = std::min(lo, k.b.lo[a]);
            hi = std::max(hi, k.b.hi[a]);
        }
        n.origin[a] = lo - 0.01f;
        const uint32_t e = ((f2u((hi - lo + 0.02f) / 255.f) >> 23) & 0xFFu) + 1u;
        n.exps[a] = (uint8_t)e;
        for(size_t k = 0; k < c.size(); ++k)
        {
            n.qlo[a][k] = (uint8_t)std::floor((c[k].b.lo[a] - 0.005f - n.origin[a]) / exp_scale(e));
            n.qhi[a][k] = (uint8_t)std::min(255.f, std::ceil((c[k].b.hi[a] + 0.005f - n.origin[a]) / exp_scale(e)));
        }
    }
    for(size_t k = 0; k < c.size(); ++k) n.child[k] = c[k].word;
    return n;
}

int main()
{
    std::mt19937 rng(7);
    auto uniform = [&](float lo, float hi) { return lo + (hi - lo) * (float)(rng() >> 8) * 0x1p-24f; };
    // a mesh of 16 random triangles around the origin: two inner nodes of four leaves of two
    std::vector<tri_rec> tris(16);
    std::vector<child> leaves;
    for(uint32_t t = 0; t < 16; ++t)
    {
        float p[9];
        box b{{9, 9, 9}, {-9, -9, -9}};
        for(int k = 0; k < 9; ++k)
        {
            p[k] = uniform(-0.5f, 0.5f);
            b.lo[k % 3] = std::min(b.lo[k % 3], p[k]);
            b.hi[k % 3] = std::max(b.hi[k % 3], p[k]);
        }
        std::memset(&tris[t], 0, sizeof(tri_rec));
        for(int k = 0; k < 3; ++k)
        {
            tris[t].v[k] = p[k];
            tris[t].v[3 + k] = p[3 + k] - p[k];
            tris[t].v[6 + k] = p[6 + k] - p[k];
        }
        tris[t].prim = t;
        if(t & 1u)
        {
            for(int a = 0; a < 3; ++a)
            {
                leaves.back().b.lo[a] = std::min(leaves.back().b.lo[a], b.lo[a]);
                leaves.back().b.hi[a] = std::max(leaves.back().b.hi[a], b.hi[a]);
            }
        }
        else
            leaves.push_back({b, LEAF_BIT | (1u << 27) | t});
    }
    const box unit{{-0.5f, -0.5f, -0.5f}, {0.5f, 0.5f, 0.5f}};
    const std::vector<child> halves[2] = {{leaves.begin(), leaves.begin() + 4}, {leaves.begin() + 4, leaves.end()}};
    std::vector<node8> mesh = {make_node({{unit, 1u}, {unit, 2u}}), make_node(halves[0]), make_node(halves[1])};
    const blas_ref blas{mesh.data(), tris.data(), 16u, 0u};
    // top levels of leaves with 16, 9, 8, 2 and 1 instances
    const uint32_t counts[5] = {16, 9, 8, 2, 1};
    std::vector<inst_rec> inst;
    std::vector<float4> boxes;
    std::vector<child> top;
    for(uint32_t c: counts)
    {
        box b{{99, 99, 99}, {-99, -99, -99}};
        const uint32_t first = (uint32_t)inst.size();
        for(uint32_t k = 0; k < c; ++k)
        {
            inst_rec r;
            std::memset(&r, 0, sizeof(r));
            const float at[3] = {uniform(-1.5f, 1.5f), uniform(-1.5f, 1.5f), uniform(-1.5f, 1.5f)};
            for(int a = 0; a < 3; ++a)
            {
                r.w2o[5 * a] = r.o2w[5 * a] = 1.f;
                r.w2o[4 * a + 3] = -at[a];
                r.o2w[4 * a + 3] = at[a];
                b.lo[a] = std::min(b.lo[a], at[a] - 0.51f);
                b.hi[a] = std::max(b.hi[a], at[a] + 0.51f);
            }
            r.instance = (uint32_t)inst.size();
            inst.push_back(r);
            boxes.push_back(make_float4(at[0] - 0.51f, at[1] - 0.51f, at[2] - 0.51f, at[0] + 0.51f));
            boxes.push_back(make_float4(at[1] + 0.51f, at[2] + 0.51f, 0.f, 0.f));
        }
        top.push_back({b, LEAF_BIT | ((c - 1u) << 27) | first});
    }
    const std::vector<node8> tnodes = {make_node(top)};

    int hits = 0, single = 0, wrong = 0;
    for(int round = 0; round < 200; ++round)
    {
        float o[4][3], d[4][3], m[4][3]; // m: directions towards the mesh
        for(int g = 0; g < 4; ++g)
            for(int a = 0; a < 3; ++a)
            {
                o[g][a] = uniform(-3.f, 3.f);
                d[g][a] = uniform(-1.f, 1.f) - 0.3f * o[g][a];
                m[g][a] = uniform(-1.f, 1.f) - o[g][a];
            }
        // the lanes in order, backwards, and at random
        int order[LANES];
        for(int l = 0; l < LANES; ++l) order[l] = round % 3 == 1 ? LANES - 1 - l : l;
        if(round % 3 == 2) std::shuffle(order, order + LANES, rng);
        tlas_result got[2][LANES];
        static uint2 stack[4][TL_GROUP_SMALL_STACK + 1];
        auto trace = [&](int l, auto any) {
            constexpr bool ANY = decltype(any)::value;
            const int g = l / GROUP_LANES;
            got[ANY][l] = trace_tlas_group<ANY, TL_GROUP_SMALL_STACK>(true, tnodes.data(), inst.data(), boxes.data(), &blas,
                                                                      o[g][0], o[g][1], o[g][2], 0.f, d[g][0], d[g][1],
                                                                      d[g][2], 1e30f, CULL_NONE, stack[g]);
        };
        run_warp(order, [&](int l) { trace(l, std::false_type{}); });
        run_warp(order, [&](int l) { trace(l, std::true_type{}); });
        trace_result one[2][LANES];
        auto trace_one = [&](int l, auto any) {
            constexpr bool ANY = decltype(any)::value;
            const int g = l / GROUP_LANES;
            one[ANY][l] = trace_group<ANY, TL_GROUP_SMALL_STACK>(true, mesh.data(), tris.data(), o[g][0], o[g][1], o[g][2],
                                                                 0.f, m[g][0], m[g][1], m[g][2], 1e30f, CULL_NONE,
                                                                 stack[g], nullptr);
        };
        run_warp(order, [&](int l) { trace_one(l, std::false_type{}); });
        run_warp(order, [&](int l) { trace_one(l, std::true_type{}); });
        for(int l = 0; l < LANES; ++l)
        {
            const int g = l / GROUP_LANES;
            const tlas_result want =
                    trace_tlas<false>(tnodes.data(), inst.data(), boxes.data(), &blas, o[g][0], o[g][1], o[g][2], 0.f, d[g][0],
                                      d[g][1], d[g][2], 1e30f, CULL_NONE);
            const tlas_result &h = got[0][l];
            hits += want.prim != VKG_MISS;
            wrong += h.prim != want.prim || h.inst != want.inst || h.t != want.t || h.u != want.u || h.v != want.v ||
                     got[1][l].occluded != (want.prim != VKG_MISS);
            unsigned long long visits = 0, tests = 0;
            const trace_result w = trace_ray<false, false, TL_GROUP_SMALL_STACK>(
                    mesh.data(), tris.data(), o[g][0], o[g][1], o[g][2], 0.f, m[g][0], m[g][1], m[g][2], 1e30f, CULL_NONE,
                    visits, tests, nullptr);
            const trace_result &s = one[0][l];
            single += w.prim != VKG_MISS;
            wrong += s.prim != w.prim || s.t != w.t || s.u != w.u || s.v != w.v ||
                     one[1][l].occluded != (w.prim != VKG_MISS);
        }
    }
    std::printf("%d lanes with a hit in the scene, %d in the mesh, %d wrong\n", hits, single, wrong);
    return hits > 1000 && single > 1000 && wrong == 0 ? 0 : 1;
}
