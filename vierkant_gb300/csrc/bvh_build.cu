// GPU LBVH build collapsed to an 8-wide quantised BVH.
//
// Replaces the reference's driver-built bottom-level acceleration structure
// (RayBuilder::create_mesh_structures, src/RayBuilder.cpp:98-300, vkCmdBuildAccelerationStructuresKHR
// at :274) and its compaction copy (:305-356). The reference's BVH is opaque; this one is fully
// specified so that every stage can be compared bit-for-bit with the CPU statement of the same
// algorithm:
//   k_tri_boxes    triangle boxes + scene box (order-independent min/max atomics)
//   k_morton       30-bit Morton code of each box centre over the scene box
//   k_radix_*      stable LSD radix sort of (code, triangle id), 8 bits per pass
//   k_karras       Karras 2012 radix tree (equal codes split by index)
//   k_refit        bottom-up boxes, second arriving child finishes the parent
//   k_topology     breadth-first collapse to 8-wide nodes: which BVH2 nodes become children, numbering
//   k_quantise     the nodes' boxes (8 bits a side) and child words, eight lanes per node
//   k_tri_records  48-byte triangle records (v0, e1, e2, id) in sorted order
// Data layout in HBM: nodes (96 B each) and triangle records (48 B each) are contiguous arrays read
// with 16-byte vector loads by the traversal kernels.
#include "internal.hpp"
#include "radix_sort.cuh"
#include "tc.cuh"

#include <algorithm>
#include <cstring>
#include <mutex>
#include <vector>

namespace vkg
{
namespace
{


struct box6
{
    float lo[3], hi[3];
};

// ordered-uint encoding: monotone for every float, so min/max atomics on it are exact
__device__ __forceinline__ uint32_t fenc(float f)
{
    uint32_t b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float fdec(uint32_t u) { return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u); }

// errors reported by the build kernels
enum : uint32_t
{
    BUILD_ERR_INDEX = 1u,    // an index >= num_vertices (triangles) / a BLAS index >= num_blas (instances)
    BUILD_ERR_CAPACITY = 2u, // node capacity exceeded
    BUILD_ERR_SINGULAR = 4u, // an instance transform that cannot be inverted
    BUILD_ERR_WAIT = 8u,     // a grid barrier of k_topology was not reached in time
};

// an internal node of the binary radix tree: what the collapse reads of it, in one 16-byte load
struct alignas(16) bvh2_node
{
    uint32_t left, right; // LEAF_BIT | sorted position, or internal node
    float area;           // half the surface area of its box (written by k_refit)
    uint32_t count;       // primitives below it
};

__global__ void k_tri_boxes(const float *__restrict__ xyz, uint32_t nv, const uint32_t *__restrict__ idx, uint32_t n,
                            box6 *__restrict__ tbox, uint32_t *__restrict__ scene_enc, uint32_t *__restrict__ err)
{
    __shared__ uint32_t s_lo[3], s_hi[3];
    if(threadIdx.x < 3)
    {
        s_lo[threadIdx.x] = fenc(__int_as_float(0x7f800000));  // +inf
        s_hi[threadIdx.x] = fenc(__int_as_float(0xff800000));  // -inf
    }
    __syncthreads();
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if(i < n)
    {
        box6 b;
        for(int a = 0; a < 3; ++a)
        {
            b.lo[a] = __int_as_float(0x7f800000);
            b.hi[a] = __int_as_float(0xff800000);
        }
        for(int k = 0; k < 3; ++k)
        {
            uint32_t vi = __ldg(&idx[3 * (size_t)i + k]);
            if(vi >= nv)
            {
                atomicOr(err, BUILD_ERR_INDEX);
                vi = 0;
            }
            for(int a = 0; a < 3; ++a)
            {
                float p = __ldg(&xyz[3 * (size_t)vi + a]);
                b.lo[a] = fminf(b.lo[a], p);
                b.hi[a] = fmaxf(b.hi[a], p);
            }
        }
        tbox[i] = b;
        for(int a = 0; a < 3; ++a)
        {
            atomicMin(&s_lo[a], fenc(b.lo[a]));
            atomicMax(&s_hi[a], fenc(b.hi[a]));
        }
    }
    __syncthreads();
    if(threadIdx.x < 3)
    {
        atomicMin(&scene_enc[threadIdx.x], s_lo[threadIdx.x]);
        atomicMax(&scene_enc[3 + threadIdx.x], s_hi[threadIdx.x]);
    }
}

__device__ __forceinline__ void scene_box(const uint32_t *scene_enc, float lo[3], float hi[3])
{
    for(int a = 0; a < 3; ++a)
    {
        lo[a] = fdec(scene_enc[a]);
        hi[a] = fdec(scene_enc[3 + a]);
    }
}

__global__ void k_morton(const box6 *__restrict__ tbox, uint32_t n, const uint32_t *__restrict__ scene_enc,
                         uint32_t *__restrict__ keys, uint32_t *__restrict__ vals, uint32_t *__restrict__ morton_out)
{
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= n) return;
    float lo[3], hi[3];
    scene_box(scene_enc, lo, hi);
    box6 b = tbox[i];
    uint32_t q[3];
    for(int a = 0; a < 3; ++a)
    {
        float e = fsub(hi[a], lo[a]);
        float scale = e > 0.f ? fdiv(1024.0f, e) : 0.f;
        float c = fmul(fadd(b.lo[a], b.hi[a]), 0.5f);
        float f = fmul(fsub(c, lo[a]), scale);
        uint32_t v = f > 0.f ? __float2uint_rz(f) : 0u;
        q[a] = v > 1023u ? 1023u : v;
    }
    uint32_t code = (expand10(q[0]) << 2) | (expand10(q[1]) << 1) | expand10(q[2]);
    keys[i] = code;
    vals[i] = i;
    morton_out[i] = code;
}

__global__ void k_karras(const uint32_t *__restrict__ codes, uint32_t n, bvh2_node *__restrict__ tree,
                         uint32_t *__restrict__ first, uint32_t *__restrict__ iparent, uint32_t *__restrict__ lparent)
{
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= (int64_t)n - 1) return;
    const int64_t nn = n;
    int d = (kdelta(codes, nn, i, i + 1) - kdelta(codes, nn, i, i - 1)) >= 0 ? 1 : -1;
    int dmin = kdelta(codes, nn, i, i - d);
    int64_t lmax = 2;
    while(kdelta(codes, nn, i, i + lmax * d) > dmin) lmax *= 2;
    int64_t l = 0;
    for(int64_t t = lmax / 2; t >= 1; t /= 2)
        if(kdelta(codes, nn, i, i + (l + t) * d) > dmin) l += t;
    int64_t j = i + l * d;
    int dnode = kdelta(codes, nn, i, j);
    int64_t s = 0, t = l;
    do
    {
        t = (t + 1) / 2;
        if(kdelta(codes, nn, i, i + (s + t) * d) > dnode) s += t;
    } while(t > 1);
    int64_t gamma = i + s * d + (d < 0 ? -1 : 0);
    int64_t lo = i < j ? i : j, hi = i < j ? j : i;
    uint32_t lc = (lo == gamma) ? (LEAF_BIT | (uint32_t)gamma) : (uint32_t)gamma;
    uint32_t rc = (hi == gamma + 1) ? (LEAF_BIT | (uint32_t)(gamma + 1)) : (uint32_t)(gamma + 1);
    *reinterpret_cast<uint4 *>(&tree[i]) = make_uint4(lc, rc, 0u, (uint32_t)(hi - lo) + 1u);
    first[i] = (uint32_t)lo;
    if(lc & LEAF_BIT) lparent[lc & ~LEAF_BIT] = (uint32_t)i;
    else iparent[lc] = (uint32_t)i;
    if(rc & LEAF_BIT) lparent[rc & ~LEAF_BIT] = (uint32_t)i;
    else iparent[rc] = (uint32_t)i;
}

__global__ void k_gather_leaf_boxes(const box6 *__restrict__ tbox, const uint32_t *__restrict__ sorted, uint32_t n,
                                    box6 *__restrict__ lbox)
{
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if(i < n) lbox[i] = tbox[sorted[i]];
}

__device__ __forceinline__ box6 load_box_cg(const box6 *p)
{
    const float *f = reinterpret_cast<const float *>(p);
    box6 b;
    for(int a = 0; a < 3; ++a)
    {
        b.lo[a] = __ldcg(f + a);
        b.hi[a] = __ldcg(f + 3 + a);
    }
    return b;
}

__device__ __forceinline__ float box_area(const box6 &b)
{
    float dx = fsub(b.hi[0], b.lo[0]), dy = fsub(b.hi[1], b.lo[1]), dz = fsub(b.hi[2], b.lo[2]);
    return fadd(fadd(fmul(dx, dy), fmul(dy, dz)), fmul(dz, dx));
}

// Bottom-up boxes: the second child to arrive at a node finishes it and goes on with its own box in
// registers. Bound by the latency of its steps, one atomic and one sibling box per level of the tree: a
// node's children and parent are fetched while the atomic is under way, and the atomic itself orders the
// boxes (two fences and both children's boxes a level took 102 us for 522,242 triangles, now 69).
__global__ void k_refit(const uint32_t *__restrict__ lparent, const uint32_t *__restrict__ iparent, bvh2_node *tree,
                        const box6 *__restrict__ lbox, box6 *ibox, uint32_t *visits, uint32_t n)
{
    const uint32_t leaf = blockIdx.x * blockDim.x + threadIdx.x;
    if(leaf >= n || n < 2) return;
    uint32_t p = lparent[leaf], self = LEAF_BIT | leaf;
    box6 u = lbox[leaf];
    // bounded: a path to the root has at most n - 1 internal nodes
    for(uint32_t guard = 0; guard < n; ++guard)
    {
        const uint2 lr = *reinterpret_cast<const uint2 *>(&tree[p]);
        const uint32_t up = p ? iparent[p] : 0u;
        uint32_t arrived;
        asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(arrived) : "l"(visits + p) : "memory");
        if(arrived == 0u) return; // first arrival: the sibling finishes p
        const uint32_t sib = lr.x == self ? lr.y : lr.x;
        const box6 o = (sib & LEAF_BIT) ? lbox[sib & ~LEAF_BIT] : load_box_cg(&ibox[sib]);
        for(int k = 0; k < 3; ++k)
        {
            u.lo[k] = fminf(u.lo[k], o.lo[k]);
            u.hi[k] = fmaxf(u.hi[k], o.hi[k]);
        }
        float *dst = reinterpret_cast<float *>(&ibox[p]);
        for(int k = 0; k < 3; ++k)
        {
            __stcg(dst + k, u.lo[k]);
            __stcg(dst + 3 + k, u.hi[k]);
        }
        tree[p].area = box_area(u);
        if(p == 0) return;
        self = p;
        p = up;
    }
}

// ---- breadth-first collapse to 8-wide nodes (deterministic numbering) -----------------------------
// how long a grid barrier waits for the other blocks (they are all resident, so it never runs out in a build);
// `absent`: arrivals it expects beyond the grid's, which never come (vkg_diag_build_timeout)
struct grid_wait
{
    uint64_t limit_ns = 4000000000ull;
    uint32_t absent = 0;
};
constexpr uint32_t GRID_WAIT_TRIES = 1u << 26; // and at most so many looks

struct collapse_args
{
    const bvh2_node *tree;
    const uint32_t *first;
    const box6 *ibox, *lbox;
    uint32_t n, leaf_max, capacity;
    const uint32_t *scene_enc;
    uint32_t *node_ref;  // [capacity] BVH2 reference of each 8-wide node
    node8 *nodes;        // [capacity]
    uint32_t *out_info;  // [0] num_nodes, [1] depth, [2] error flags, [3] grid barrier (zero at launch)
    uint32_t *block_sum; // [grid] children of a block's nodes in the current level
    float *out_margin;
    grid_wait wait;
};

__device__ __forceinline__ uint32_t ref_count(const collapse_args &A, uint32_t r)
{
    return (r & LEAF_BIT) ? 1u : A.tree[r].count;
}

// Grid barrier of a cooperative launch, the `barrier`-th of the kernel: every block adds one to *arrived. false
// when the others did not arrive within the limit, which it reports to them.
__device__ bool grid_barrier(uint32_t *arrived, uint32_t barrier, uint32_t *err, const grid_wait &wait)
{
    __shared__ uint32_t s_ok;
    __syncthreads();
    if(threadIdx.x == 0)
    {
        const uint32_t target = gridDim.x * barrier + wait.absent;
        s_ok = 1u;
        __threadfence();
        atomicAdd(arrived, 1u);
        uint64_t start = 0;
        for(uint32_t tries = 0; *reinterpret_cast<volatile uint32_t *>(arrived) < target; ++tries)
        {
            // (the clock is read now and then: a look at the counter is what the barrier's latency consists of)
            bool out = tries > GRID_WAIT_TRIES || (*reinterpret_cast<volatile uint32_t *>(err) & BUILD_ERR_WAIT);
            if((tries & 255u) == 255u)
            {
                const uint64_t now = tc::global_ns();
                if(!start) start = now;
                out = out || now - start > wait.limit_ns;
            }
            if(!out) continue;
            atomicOr(err, BUILD_ERR_WAIT);
            s_ok = 0u;
            break;
        }
        __threadfence();
    }
    __syncthreads();
    return s_ok != 0u;
}

constexpr int COLLAPSE_THREADS = 512;
// nodes per block below which further blocks would only add to the barriers
constexpr uint32_t COLLAPSE_PRIMS_PER_BLOCK = 2048;

// inclusive scan of x over the block; `total` receives the block's sum
__device__ __forceinline__ uint32_t block_scan(uint32_t x, uint32_t *s_warp, uint32_t &total)
{
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    for(int o = 1; o < 32; o <<= 1)
    {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if(lane >= (uint32_t)o) x += y;
    }
    __syncthreads(); // s_warp may still be read for the call before
    if(lane == 31) s_warp[warp] = x;
    __syncthreads();
    uint32_t before = 0;
    total = 0;
    for(uint32_t w = 0; w < COLLAPSE_THREADS / 32; ++w)
    {
        const uint32_t v = s_warp[w];
        before += w < warp ? v : 0u;
        total += v;
    }
    return before + x;
}

// Level by level, every 8-wide node of the level opens its BVH2 node until eight children are found or
// only leaves are left (the largest box first); the internal children of a level, in node and slot
// order, are the next level's nodes. A level's nodes are split over the blocks in contiguous runs;
// one scan over the blocks' child counts numbers the next level exactly as one block would.
// Between this kernel and k_quantise a node holds: child[] = its BVH2 references, origin[0] = index
// of its first internal child, origin[1] = bit mask of the internal children, nchild.
// Bound by the latency of the dependent loads of a node's opening (7 steps) and of two grid barriers
// a level. One block did all of this and the quantisation before, 4.76 ms for 522,242 triangles.
__global__ void __launch_bounds__(COLLAPSE_THREADS) k_topology(collapse_args A)
{
    __shared__ uint32_t s_warp[COLLAPSE_THREADS / 32];
    const uint32_t tid = threadIdx.x;
    if(blockIdx.x == 0 && tid == 0)
    {
        float lo[3], hi[3];
        scene_box(A.scene_enc, lo, hi);
        float ext = 0.f, amax = 0.f;
        for(int a = 0; a < 3; ++a)
        {
            ext = fmaxf(ext, fsub(hi[a], lo[a]));
            amax = fmaxf(amax, fmaxf(fabsf(lo[a]), fabsf(hi[a])));
        }
        *A.out_margin = fmul(fmaxf(ext, amax), 3.0517578125e-05f); // 2^-15
        __stcg(&A.node_ref[0], (A.n == 1) ? (LEAF_BIT | 0u) : 0u);
    }
    __syncthreads();
    uint32_t begin = 0, end = 1, depth = 0, barriers = 0, err = 0;
    while(begin < end)
    {
        ++depth;
        // whole rounds of the block per block: a level of few nodes stays with few blocks
        const uint32_t rounds = (end - begin + COLLAPSE_THREADS - 1) / COLLAPSE_THREADS;
        const uint32_t per = (rounds + gridDim.x - 1) / gridDim.x * COLLAPSE_THREADS;
        const uint32_t lo = min(begin + blockIdx.x * per, end), hi = min(lo + per, end);
        uint32_t carry = 0;
        for(uint32_t base = lo; base < hi; base += COLLAPSE_THREADS)
        {
            const uint32_t ni = base + tid;
            const bool active = ni < hi;
            uint32_t slot[8], ns = 0, inner = 0;
            if(active)
            {
                // per slot: its reference, the box area (-1: not to be opened) and its children
                float area[8];
                uint32_t left[8], right[8];
                const uint32_t r = __ldcg(&A.node_ref[ni]);
#pragma unroll
                for(int k = 0; k < 8; ++k)
                {
                    slot[k] = left[k] = right[k] = 0u;
                    area[k] = -1.f;
                }
                auto put = [&](int at, uint32_t ref) {
                    uint4 v = make_uint4(0u, 0u, __float_as_uint(-1.f), 1u);
                    if(!(ref & LEAF_BIT)) v = *reinterpret_cast<const uint4 *>(&A.tree[ref]);
                    const bool open = v.w > A.leaf_max;
#pragma unroll
                    for(int k = 0; k < 8; ++k)
                        if(k == at)
                        {
                            slot[k] = ref;
                            left[k] = v.x;
                            right[k] = v.y;
                            area[k] = open ? __uint_as_float(v.z) : -1.f;
                        }
                    inner = (inner & ~(1u << at)) | (open ? 1u << at : 0u);
                };
                // (only the root of a single primitive is a leaf)
                if(r & LEAF_BIT) put((int)ns++, r);
                else
                {
                    const uint2 lr = *reinterpret_cast<const uint2 *>(&A.tree[r]);
                    put(0, lr.x);
                    put(1, lr.y);
                    for(ns = 2; ns < 8; ++ns)
                    {
                        int best = -1;
                        float best_area = -1.f;
                        uint32_t bl = 0, br = 0;
#pragma unroll
                        for(int k = 0; k < 8; ++k)
                            if(area[k] > best_area)
                            {
                                best_area = area[k];
                                best = k;
                                bl = left[k];
                                br = right[k];
                            }
                        if(best < 0) break;
                        put(best, bl);
                        put((int)ns, br);
                    }
                }
            }
            uint32_t total;
            const uint32_t nint = __popc(inner), incl = block_scan(nint, s_warp, total);
            if(active)
            {
                node8 *nd = A.nodes + ni;
                uint4 *w = reinterpret_cast<uint4 *>(nd);
                w[0] = make_uint4(carry + incl - nint, inner, 0u, ns << 24);
                w[4] = make_uint4(slot[0], slot[1], slot[2], slot[3]);
                w[5] = make_uint4(slot[4], slot[5], slot[6], slot[7]);
            }
            carry += total;
        }
        uint32_t before = 0, next = 0; // children of the blocks before this one / of all
        if(gridDim.x > 1)
        {
            if(tid == 0) __stcg(&A.block_sum[blockIdx.x], carry);
            if(!grid_barrier(&A.out_info[3], ++barriers, &A.out_info[2], A.wait)) return;
            uint32_t b = 0, t = 0;
            for(uint32_t k = tid; k < gridDim.x; k += COLLAPSE_THREADS)
            {
                const uint32_t v = __ldcg(&A.block_sum[k]);
                b += k < blockIdx.x ? v : 0u;
                t += v;
            }
            block_scan(b, s_warp, before);
            block_scan(t, s_warp, next);
        }
        else
        {
            next = carry;
            __syncthreads();
        }
        const uint32_t room = A.capacity - min(end, A.capacity);
        if(next > room)
        {
            err = BUILD_ERR_CAPACITY;
            end += next;
            break;
        }
        for(uint32_t ni = lo + tid; ni < hi; ni += COLLAPSE_THREADS)
        {
            uint32_t *w = reinterpret_cast<uint32_t *>(A.nodes + ni);
            const uint32_t c0 = end + before + w[0];
            uint32_t c = c0;
            for(uint32_t m = w[1]; m; m &= m - 1u) __stcg(&A.node_ref[c++], w[16 + __ffs(m) - 1]);
            w[0] = c0;
        }
        begin = end;
        end += next;
        if(gridDim.x > 1 && begin < end)
        {
            if(!grid_barrier(&A.out_info[3], ++barriers, &A.out_info[2], A.wait)) return;
        }
        else
            __syncthreads();
    }
    if(blockIdx.x == 0 && tid == 0)
    {
        A.out_info[0] = end;
        A.out_info[1] = depth;
        if(err) atomicOr(&A.out_info[2], err);
    }
}

// The nodes' quantised boxes and child words. Eight lanes per node, one child each: the child boxes are
// read side by side, the node's box is a three-step shuffle reduction, and every field of the node is
// written by neighbouring lanes.
__global__ void __launch_bounds__(256) k_quantise(collapse_args A)
{
    if(A.out_info[2]) return;
    const uint32_t num = A.out_info[0], lane = threadIdx.x & 31u, k = lane & 7u;
    const float m = *A.out_margin;
    const uint32_t warps = gridDim.x * (blockDim.x / 32u);
    for(uint32_t n0 = 4u * (blockIdx.x * (blockDim.x / 32u) + (threadIdx.x >> 5)); n0 < num; n0 += 4u * warps)
    {
        const uint32_t ni = n0 + (lane >> 3);
        const bool active = ni < num;
        uint32_t ref = 0, ns = 0, inner = 0, c0 = 0;
        if(active)
        {
            const uint32_t *w = reinterpret_cast<const uint32_t *>(A.nodes + ni);
            c0 = w[0];
            inner = w[1];
            ns = w[3] >> 24;
            ref = w[16 + k];
        }
        const bool valid = k < ns;
        float lo[3], hi[3], nlo[3], nhi[3];
        box6 b;
        if(valid) b = (ref & LEAF_BIT) ? A.lbox[ref & ~LEAF_BIT] : A.ibox[ref];
#pragma unroll
        for(int a = 0; a < 3; ++a)
        {
            lo[a] = valid ? fsub(b.lo[a], m) : __int_as_float(0x7f800000);
            hi[a] = valid ? fadd(b.hi[a], m) : __int_as_float(0xff800000);
            nlo[a] = lo[a];
            nhi[a] = hi[a];
#pragma unroll
            for(int o = 1; o < 8; o <<= 1)
            {
                nlo[a] = fminf(nlo[a], __shfl_xor_sync(0xffffffffu, nlo[a], o));
                nhi[a] = fmaxf(nhi[a], __shfl_xor_sync(0xffffffffu, nhi[a], o));
            }
        }
        __syncwarp(); // every lane has read the node's words
        if(!active) continue;
        uint8_t *out = reinterpret_cast<uint8_t *>(A.nodes + ni);
        uint32_t exps = 0;
#pragma unroll
        for(int a = 0; a < 3; ++a)
        {
            const float xq = fdiv(fsub(nhi[a], nlo[a]), 255.0f);
            uint32_t e = ((__float_as_uint(xq) >> 23) & 0xFFu) + 1u;
            if(e > 254u) e = 254u;
            exps |= e << (8 * a);
            const float inv_s = exp_scale(254u - e);
            uint8_t ql = 0, qh = 0;
            if(valid)
            {
                const float fl = floorf(fmul(fsub(lo[a], nlo[a]), inv_s));
                const float fh = ceilf(fmul(fsub(hi[a], nlo[a]), inv_s));
                ql = (uint8_t)(fl < 0.f ? 0.f : (fl > 255.f ? 255.f : fl));
                qh = (uint8_t)(fh < 0.f ? 0.f : (fh > 255.f ? 255.f : fh));
            }
            out[16 + 8 * a + k] = ql;
            out[40 + 8 * a + k] = qh;
        }
        uint32_t word = 0u;
        if(valid)
        {
            if((inner >> k) & 1u) word = c0 + __popc(inner & ((1u << k) - 1u));
            else
            {
                const uint32_t cnt = ref_count(A, ref), at = (ref & LEAF_BIT) ? (ref & ~LEAF_BIT) : A.first[ref];
                word = LEAF_BIT | ((cnt - 1u) << 27) | at;
            }
        }
        reinterpret_cast<uint32_t *>(out)[16 + k] = word;
        if(k == 0)
            *reinterpret_cast<uint4 *>(out) = make_uint4(__float_as_uint(nlo[0]), __float_as_uint(nlo[1]),
                                                         __float_as_uint(nlo[2]), exps | (ns << 24));
    }
}

__global__ void k_tri_records(const float *__restrict__ xyz, uint32_t nv, const uint32_t *__restrict__ idx,
                              const uint32_t *__restrict__ sorted, uint32_t n, tri_rec *__restrict__ out)
{
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= n) return;
    uint32_t p = sorted[i];
    float v[3][3];
    for(int k = 0; k < 3; ++k)
    {
        uint32_t vi = idx[3 * (size_t)p + k];
        if(vi >= nv) vi = 0;
        for(int a = 0; a < 3; ++a) v[k][a] = xyz[3 * (size_t)vi + a];
    }
    tri_rec r;
    for(int a = 0; a < 3; ++a)
    {
        r.v[a] = v[0][a];
        r.v[3 + a] = fsub(v[1][a], v[0][a]);
        r.v[6 + a] = fsub(v[2][a], v[0][a]);
    }
    r.prim = p;
    r.pad[0] = r.pad[1] = 0u;
    out[i] = r;
}

template<typename T>
cudaError_t dalloc(vkg_ctx *ctx, T **p, size_t count, cudaStream_t s)
{
    return ctx_alloc(ctx, reinterpret_cast<void **>(p), count * sizeof(T) + 16, s);
}

// hands out 256-byte aligned pieces of one allocation (of no allocation yet: only adds up their sizes)
struct arena
{
    uintptr_t base = 0;
    size_t used = 0;
    template<typename T>
    void take(T *&p, size_t count)
    {
        p = reinterpret_cast<T *>(base + used);
        used += (count * sizeof(T) + 255) & ~size_t(255);
    }
};

// what a build starts from: [0..5] the empty scene box (ordered uints: +inf, -inf), [6] error bits of the
// primitives, [8..10] the collapse's info, [11] its grid barrier, [12] the margin, [13] half the surface areas of the
// instances' boxes (0 for triangles)
__global__ void k_build_init(uint32_t *__restrict__ visits, uint32_t n, uint32_t *__restrict__ small)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if(i < n) visits[i] = 0u;
    if(i < 16) small[i] = i < 3 ? 0xFF800000u : (i < 6 ? 0x007FFFFFu : 0u);
}

// ---- instances (two-level BVH) -------------------------------------------------------------------
struct blas_box
{
    float lo[3], hi[3];
    uint32_t num_tris, pad;
    const node8 *nodes; // the BLAS's nodes: its upper levels give a tighter instance box than its bounds
};

// corner of child k of a node (words w): coordinate c, the box's high side or its low one. Layout
// (traverse.cuh, node_keys): origin in words 0-2, scales in 3, lo x / y / z in words 4-5 / 6-7 / 8-9, hi in 10-15
__device__ __forceinline__ uint32_t child_quant(const uint32_t *w, int k, int c, bool high)
{
    return (w[(high ? 10 : 4) + 2 * c + (k >> 2)] >> (8 * (k & 3))) & 0xFFu;
}
__device__ __forceinline__ float child_scale(const uint32_t *w, int c) { return exp_scale((w[3] >> (8 * c)) & 0xFFu); }

// box slot s (0..63) of a BLAS, two levels below its root: child s & 7 of root child s >> 3, or a leaf of the
// root at s & 7 = 0. The words of the node that holds the box and its child there; false if there is none
__device__ __forceinline__ bool box_slot(const node8 *nodes, uint32_t s, const uint32_t *&w, int &k)
{
    w = reinterpret_cast<const uint32_t *>(nodes);
    k = (int)(s >> 3);
    if((uint32_t)k >= w[3] >> 24) return false;
    const uint32_t c = w[16 + k];
    if(c & LEAF_BIT) return (s & 7u) == 0u;
    w = reinterpret_cast<const uint32_t *>(nodes + c);
    k = (int)(s & 7u);
    return (uint32_t)k < w[3] >> 24;
}

// world -> object transform of an object -> world 3x4 transform: inverse of the 3x3 part by the
// adjugate in double precision, translation -A^-1 t, rounded to float once. false if singular.
__device__ __forceinline__ bool invert_3x4(const float *m, float *inv)
{
    const double a = m[0], b = m[1], c = m[2], d = m[4], e = m[5], f = m[6], g = m[8], h = m[9], i = m[10];
    const double A = __dsub_rn(__dmul_rn(e, i), __dmul_rn(f, h));
    const double B = __dsub_rn(__dmul_rn(f, g), __dmul_rn(d, i));
    const double C = __dsub_rn(__dmul_rn(d, h), __dmul_rn(e, g));
    const double det = __dadd_rn(__dadd_rn(__dmul_rn(a, A), __dmul_rn(b, B)), __dmul_rn(c, C));
    if(!(fabs(det) > 1e-30) || !isfinite(det)) return false;
    const double r = 1.0 / det;
    const double M[9] = {A, __dsub_rn(__dmul_rn(c, h), __dmul_rn(b, i)), __dsub_rn(__dmul_rn(b, f), __dmul_rn(c, e)),
                         B, __dsub_rn(__dmul_rn(a, i), __dmul_rn(c, g)), __dsub_rn(__dmul_rn(c, d), __dmul_rn(a, f)),
                         C, __dsub_rn(__dmul_rn(b, g), __dmul_rn(a, h)), __dsub_rn(__dmul_rn(a, e), __dmul_rn(b, d))};
    const double t[3] = {m[3], m[7], m[11]};
    for(int row = 0; row < 3; ++row)
    {
        double acc = 0.0;
        for(int k = 0; k < 3; ++k)
        {
            const double v = __dmul_rn(M[3 * row + k], r);
            inv[4 * row + k] = __double2float_rn(v);
            acc = __dadd_rn(acc, __dmul_rn(v, t[k]));
        }
        inv[4 * row + 3] = __double2float_rn(-acc);
    }
    return true;
}

// World boxes of the instances, one warp each: the union of the transformed boxes two levels below the
// BLAS root (a rotated mesh's own bounds would be loose: a sphere's rotated bounding cube holds up to 5x
// its volume), two of them per lane. A side of the union is the smallest (largest) of 64 sums in FP64, and
// of a box's eight corners the one whose products are all the smallest gives it, as rounding is monotone.
// The sums in FP32, with a bound of their error, leave one or a few boxes that can hold the extreme; FP64
// (two operations a clock and SM) evaluates those alone, five lanes a side.
// 20,000 instances: 68 us; 225 us with every sum in FP64.
__global__ void __launch_bounds__(256)
        k_instance_boxes(const vkg_instance *__restrict__ inst, uint32_t n, const blas_box *__restrict__ bb,
                         uint32_t nblas, box6 *__restrict__ tbox, uint32_t *__restrict__ scene_enc,
                         uint32_t *__restrict__ err, float *__restrict__ area)
{
    __shared__ uint32_t s_lo[3], s_hi[3];
    __shared__ float s_area; // half the surface areas of the block's boxes
    if(threadIdx.x == 0) s_area = 0.f;
    if(threadIdx.x < 3)
    {
        s_lo[threadIdx.x] = fenc(__int_as_float(0x7f800000));
        s_hi[threadIdx.x] = fenc(__int_as_float(0xff800000));
    }
    __syncthreads();
    const uint32_t i = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31u;
    if(i < n)
    {
        const vkg_instance I = inst[i];
        uint32_t bl = I.blas;
        if(bl >= nblas)
        {
            if(lane == 0) atomicOr(err, BUILD_ERR_INDEX);
            bl = 0;
        }
        const blas_box B = bb[bl];
        float inv[12];
        if(lane == 0 && !invert_3x4(I.transform, inv)) atomicOr(err, BUILD_ERR_SINGULAR);
        // sides 0..2: the lows, 3..5: the highs negated; lane l evaluates side l mod 6 (lanes 30, 31: none)
        const uint32_t side = lane % 6u;
        uint64_t cand = 0;
        if(B.num_tris)
        {
            float low[2][6], up[6]; // bounds of this lane's two boxes, and of the least of them from above
            bool have[2];
#pragma unroll
            for(int d = 0; d < 6; ++d) up[d] = __int_as_float(0x7f800000);
#pragma unroll
            for(int it = 0; it < 2; ++it)
            {
                const uint32_t *w;
                int k;
                have[it] = box_slot(B.nodes, lane + 32u * it, w, k);
                if(!have[it]) continue;
                float lo[3], hi[3];
#pragma unroll
                for(int c = 0; c < 3; ++c)
                {
                    const float o = __uint_as_float(w[c]), sc = child_scale(w, c);
                    lo[c] = fmaf((float)child_quant(w, k, c, false), sc, o);
                    hi[c] = fmaf((float)child_quant(w, k, c, true), sc, o);
                }
#pragma unroll
                for(int d = 0; d < 6; ++d)
                {
                    const float *T = I.transform + 4 * (d % 3);
                    float v = T[3], mag = fabsf(T[3]);
#pragma unroll
                    for(int c = 0; c < 3; ++c)
                    {
                        const float x = (T[c] < 0.f) != (d >= 3) ? hi[c] : lo[c];
                        v = fmaf(T[c], x, v);
                        mag = fmaf(fabsf(T[c]), fabsf(x), mag);
                    }
                    // at most 6 roundings of 2^-24, each of at most mag; 2^-20 also covers mag's own
                    const float e = fmaf(mag, 0x1p-20f, 0x1p-120f), key = d < 3 ? v : -v;
                    low[it][d] = key - e;
                    up[d] = fminf(up[d], key + e);
                }
            }
            __syncwarp();
#pragma unroll
            for(int d = 0; d < 6; ++d)
            {
                // a box is out if it cannot reach the least upper bound; one that is not a number stays in
                const float least = fdec(__reduce_min_sync(0xffffffffu, fenc(up[d])));
                const uint32_t m0 = __ballot_sync(0xffffffffu, have[0] && !(low[0][d] > least));
                const uint32_t m1 = __ballot_sync(0xffffffffu, have[1] && !(low[1][d] > least));
                if(side == (uint32_t)d) cand = m0 | ((uint64_t)m1 << 32);
            }
            if(lane >= 30) cand = 0;
            for(uint32_t k = lane / 6u; k; --k) cand &= cand - 1; // every fifth candidate, from the (l / 6)th on
        }
        const uint32_t axis = side % 3u;
        const bool high = side >= 3u;
        const float *T = inst[i].transform + 4 * axis;
        double best = 1e300;
        while(cand)
        {
            const uint32_t *w;
            int k;
            box_slot(B.nodes, (uint32_t)__ffsll(cand) - 1u, w, k);
            double c[3];
            for(int a = 0; a < 3; ++a)
                c[a] = (double)__uint_as_float(w[a]) +
                       (double)child_quant(w, k, a, (T[a] < 0.f) != high) * (double)child_scale(w, a);
            const double v = (double)T[0] * c[0] + (double)T[1] * c[1] + (double)T[2] * c[2] + (double)T[3];
            best = fmin(best, high ? -v : v);
            for(int t = 0; t < 5; ++t) cand &= cand - 1;
        }
        __syncwarp();
        double least = best;
        for(uint32_t d = 6; d < 30; d += 6) least = fmin(least, __shfl_sync(0xffffffffu, best, lane + d));
        // rounded outward; the collapse grows every box by its margin on top. An empty mesh: a
        // point box at the instance origin (the traversal skips it)
        const float f = !B.num_tris ? T[3] : (high ? __double2float_ru(-least) : __double2float_rd(least));
        const float g = __shfl_down_sync(0xffffffffu, f, 3) - f; // lanes 0..2: the box's extents
        const float gy = __shfl_sync(0xffffffffu, g, 1), gz = __shfl_sync(0xffffffffu, g, 2);
        if(lane == 0) atomicAdd(&s_area, g * gy + gy * gz + gz * g);
        if(lane < 6)
        {
            (high ? tbox[i].hi : tbox[i].lo)[axis] = f;
            if(high) atomicMax(&s_hi[axis], fenc(f));
            else atomicMin(&s_lo[axis], fenc(f));
        }
    }
    __syncthreads();
    if(threadIdx.x < 3)
    {
        atomicMin(&scene_enc[threadIdx.x], s_lo[threadIdx.x]);
        atomicMax(&scene_enc[3 + threadIdx.x], s_hi[threadIdx.x]);
    }
    if(threadIdx.x == 0) atomicAdd(area, s_area);
}

// instance records in leaf (sorted) order and in input order
__global__ void k_instance_records(const vkg_instance *__restrict__ inst, const uint32_t *__restrict__ sorted,
                                   uint32_t n, uint32_t nblas, const box6 *__restrict__ lbox,
                                   const float *__restrict__ margin, inst_rec *__restrict__ out,
                                   inst_rec *__restrict__ by_id, float4 *__restrict__ box)
{
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if(i >= n) return;
    const uint32_t id = sorted[i];
    const vkg_instance I = inst[id];
    inst_rec r{};
    if(!invert_3x4(I.transform, r.w2o))
        for(int k = 0; k < 12; ++k) r.w2o[k] = 0.f;
    for(int k = 0; k < 12; ++k) r.o2w[k] = I.transform[k];
    r.blas = I.blas < nblas ? I.blas : 0u;
    r.instance = id;
    r.material = I.material;
    out[i] = r;
    by_id[id] = r;
    const box6 b = lbox[i];
    const float m = *margin;
    box[2 * (size_t)i] = make_float4(fsub(b.lo[0], m), fsub(b.lo[1], m), fsub(b.lo[2], m), fadd(b.hi[0], m));
    box[2 * (size_t)i + 1] = make_float4(fadd(b.hi[1], m), fadd(b.hi[2], m), 0.f, 0.f);
}

// both kernels of the collapse. max_blocks 1 keeps to plain launches; more blocks need a cooperative
// one, as they wait for each other (all of them fit on the device at once: one per SM)
cudaError_t launch_collapse(const collapse_args &A, uint32_t max_blocks, cudaStream_t st)
{
    uint32_t grid = std::min(max_blocks, (A.n + COLLAPSE_PRIMS_PER_BLOCK - 1) / COLLAPSE_PRIMS_PER_BLOCK);
    if(grid > 1)
    {
        void *args[] = {const_cast<collapse_args *>(&A)};
        const cudaError_t e = cudaLaunchCooperativeKernel(reinterpret_cast<const void *>(k_topology), dim3(grid),
                                                          dim3(COLLAPSE_THREADS), args, 0, st);
        if(e != cudaSuccess) return e;
    }
    else
        k_topology<<<1, COLLAPSE_THREADS, 0, st>>>(A);
    k_quantise<<<std::min((A.n + 31u) / 32u, 1216u), 256, 0, st>>>(A);
    return cudaGetLastError();
}

// The primitive-independent part of a build: make_boxes(tbox, scene_enc, err) fills the n primitive
// boxes, the scene box (ordered uints) and error bits; Morton codes, the radix sort, the Karras tree,
// the refit and the 8-wide collapse follow; make_records(sorted, lbox, margin) writes the leaf
// records in sorted order (lbox: the boxes in that order). On success bvh holds the nodes, Morton codes, sorted order, scene box, margin and depth, and
// err_bits the error bits that make_boxes raised. The caller frees bvh on failure.
template<class MakeBoxes, class MakeRecords>
vkg_status build_core(vkg_ctx *ctx, vkg_bvh *bvh, uint32_t n, uint32_t leaf_max, const grid_wait &wait, cudaStream_t st,
                      MakeBoxes make_boxes, MakeRecords make_records, uint32_t &err_bits, float &box_area)
{
    cudaEvent_t ev0, ev1;
    cudaEventCreate(&ev0);
    cudaEventCreate(&ev1);
    cudaEventRecord(ev0, st);

    // scratch, one allocation
    box6 *tbox, *lbox, *ibox;
    uint32_t *keys0, *keys1, *vals0, *vals1, *counts, *first, *iparent, *lparent, *visits, *node_ref, *block_sum, *small;
    bvh2_node *tree;
    node8 *nodes_tmp;
    const uint32_t ni = n > 1 ? n - 1 : 1;
    const uint32_t capacity = n + 8;
    arena mem;
    auto lay_out = [&]() {
        mem.used = 0;
        mem.take(tbox, n);
        mem.take(lbox, n);
        mem.take(ibox, ni);
        mem.take(keys0, n);
        mem.take(keys1, n);
        mem.take(vals0, n);
        mem.take(vals1, n);
        mem.take(counts, sort_count_words(n));
        mem.take(tree, ni);
        mem.take(first, ni);
        mem.take(iparent, ni);
        mem.take(lparent, n);
        mem.take(visits, ni);
        mem.take(node_ref, capacity);
        mem.take(nodes_tmp, capacity);
        mem.take(block_sum, (size_t)ctx->num_sms);
        mem.take(small, 16);
    };
    lay_out();
    void *scratch = nullptr;
    cudaError_t e = cudaSuccess;
    auto chk = [&](cudaError_t x) {
        if(e == cudaSuccess) e = x;
    };
    chk(ctx_alloc(ctx, &scratch, mem.used, st));
    if(e == cudaSuccess) chk(dalloc(ctx, &bvh->d_morton, n, st));
    if(e == cudaSuccess) chk(dalloc(ctx, &bvh->d_sorted, n, st));
    if(e != cudaSuccess)
    {
        if(scratch) cudaFreeAsync(scratch, st);
        cudaEventDestroy(ev0);
        cudaEventDestroy(ev1);
        cudaGetLastError();
        return set_error(ctx, VKG_ERR_OUT_OF_MEMORY, "BVH build: device allocation failed (%s)", cudaGetErrorString(e));
    }
    mem.base = reinterpret_cast<uintptr_t>(scratch);
    lay_out();
    k_build_init<<<(std::max(ni, 16u) + 255) / 256, 256, 0, st>>>(visits, ni, small);

    const int T = 256;
    const uint32_t g = (n + T - 1) / T;
    make_boxes(tbox, small, small + 6);
    k_morton<<<g, T, 0, st>>>(tbox, n, small, keys0, vals0, bvh->d_morton);
    uint32_t *kin = keys0, *kout = keys1, *vin = vals0, *vout = vals1;
    radix_sort(kin, vin, kout, vout, n, 30, counts, st);
    chk(cudaMemcpyAsync(bvh->d_sorted, vin, sizeof(uint32_t) * n, cudaMemcpyDeviceToDevice, st));
    k_gather_leaf_boxes<<<g, T, 0, st>>>(tbox, vin, n, lbox);
    if(n > 1)
    {
        k_karras<<<(ni + T - 1) / T, T, 0, st>>>(kin, n, tree, first, iparent, lparent);
        k_refit<<<g, T, 0, st>>>(lparent, iparent, tree, lbox, ibox, visits, n);
    }
    collapse_args A{tree,     first,     ibox,      lbox,      n,        leaf_max, capacity, small,
                    node_ref, nodes_tmp, small + 8, block_sum, reinterpret_cast<float *>(small + 12),
                    wait};
    chk(launch_collapse(A, (uint32_t)ctx->num_sms, st));
    make_records(static_cast<const uint32_t *>(vin), lbox, reinterpret_cast<const float *>(small + 12));
    chk(cudaGetLastError());

    uint32_t info[16];
    chk(cudaMemcpyAsync(info, small, sizeof(info), cudaMemcpyDeviceToHost, st));
    chk(cudaStreamSynchronize(st));
    if(e == cudaSuccess)
    {
        bvh->num_nodes = info[8];
        bvh->depth = info[9];
        std::memcpy(&bvh->margin, &info[12], 4);
        std::memcpy(&box_area, &info[13], 4);
        for(int a = 0; a < 3; ++a)
        {
            uint32_t lo = info[a], hi = info[3 + a];
            uint32_t lb = (lo & 0x80000000u) ? (lo & 0x7FFFFFFFu) : ~lo;
            uint32_t hb = (hi & 0x80000000u) ? (hi & 0x7FFFFFFFu) : ~hi;
            std::memcpy(&bvh->scene_min[a], &lb, 4);
            std::memcpy(&bvh->scene_max[a], &hb, 4);
        }
        chk(dalloc(ctx, &bvh->d_nodes, bvh->num_nodes, st));
        if(e == cudaSuccess)
            chk(cudaMemcpyAsync(bvh->d_nodes, nodes_tmp, sizeof(node8) * bvh->num_nodes, cudaMemcpyDeviceToDevice,
                                st));
    }
    cudaFreeAsync(scratch, st);
    cudaEventRecord(ev1, st);
    chk(cudaEventSynchronize(ev1));
    cudaEventElapsedTime(&bvh->build_ms, ev0, ev1);
    cudaEventDestroy(ev0);
    cudaEventDestroy(ev1);
    if(e != cudaSuccess) return cuda_check(ctx, e, "BVH build");
    err_bits = info[6];
    if(info[10] & BUILD_ERR_WAIT) return set_error(ctx, VKG_ERR_TIMEOUT, "BVH build: a grid barrier ran out");
    if(info[10] & BUILD_ERR_CAPACITY) return set_error(ctx, VKG_ERR_CAPACITY, "BVH build: node capacity exceeded");
    const uint32_t max_depth = (TRAVERSAL_STACK - 1) / 7 + 1;
    if(bvh->depth > max_depth)
        return set_error(ctx, VKG_ERR_CAPACITY, "BVH build: depth %u exceeds the traversal limit %u", bvh->depth,
                         max_depth);
    return VKG_OK;
}

}// namespace
}// namespace vkg

using namespace vkg;

static vkg_status bvh_build(vkg_ctx *ctx, const float *d_xyz, uint32_t num_vertices, const uint32_t *d_indices,
                            uint32_t num_tris, const vkg_bvh_build_options *opts, const grid_wait &wait, vkg_bvh **out,
                            void *stream_)
{
    if(!ctx) return VKG_ERR_INVALID_ARGUMENT;
    if(!out) return set_error(ctx, VKG_ERR_INVALID_ARGUMENT, "vkg_bvh_build: out is NULL");
    *out = nullptr;
    if(num_tris > 0 && (!d_xyz || !d_indices || num_vertices == 0))
        return set_error(ctx, VKG_ERR_INVALID_ARGUMENT, "vkg_bvh_build: NULL geometry for %u triangles", num_tris);
    if(num_tris >= MAX_TRIS)
        return set_error(ctx, VKG_ERR_CAPACITY, "vkg_bvh_build: %u triangles exceed the maximum of %u", num_tris,
                         MAX_TRIS - 1);
    uint32_t leaf_max = (opts && opts->leaf_max) ? opts->leaf_max : 2u;
    if(leaf_max > LEAF_MAX_LIMIT)
        return set_error(ctx, VKG_ERR_INVALID_ARGUMENT, "vkg_bvh_build: leaf_max %u > %u", leaf_max, LEAF_MAX_LIMIT);
    if(vkg_status s = bind_device(ctx); s != VKG_OK) return s;

    cudaStream_t st = static_cast<cudaStream_t>(stream_);
    auto *bvh = new vkg_bvh();
    bvh->device = ctx->device;
    bvh->num_tris = num_tris;
    bvh->leaf_max = leaf_max;
    if(num_tris == 0)
    {
        *out = bvh;
        return VKG_OK;
    }
    const uint32_t n = num_tris;
    if(dalloc(ctx, &bvh->d_tris, n, st) != cudaSuccess)
    {
        vkg_bvh_destroy(ctx, bvh);
        return set_error(ctx, VKG_ERR_OUT_OF_MEMORY, "vkg_bvh_build: device allocation failed");
    }
    const int T = 256;
    const uint32_t g = (n + T - 1) / T;
    uint32_t err_bits = 0;
    float box_area = 0.f;
    vkg_status s = build_core(
            ctx, bvh, n, leaf_max, wait, st,
            [&](box6 *tbox, uint32_t *scene_enc, uint32_t *err) {
                k_tri_boxes<<<g, T, 0, st>>>(d_xyz, num_vertices, d_indices, n, tbox, scene_enc, err);
            },
            [&](const uint32_t *sorted, const box6 *, const float *) {
                k_tri_records<<<g, T, 0, st>>>(d_xyz, num_vertices, d_indices, sorted, n, bvh->d_tris);
            },
            err_bits, box_area);
    if(s == VKG_OK && (err_bits & BUILD_ERR_INDEX))
        s = set_error(ctx, VKG_ERR_INVALID_ARGUMENT, "vkg_bvh_build: triangle index >= num_vertices (%u)", num_vertices);
    if(s != VKG_OK)
    {
        vkg_bvh_destroy(ctx, bvh);
        return s;
    }
    bvh->bytes = sizeof(node8) * bvh->num_nodes + sizeof(tri_rec) * n + 8 * (size_t)n;
    *out = bvh;
    return VKG_OK;
}

extern "C" vkg_status vkg_bvh_build(vkg_ctx *ctx, const float *d_xyz, uint32_t num_vertices,
                                    const uint32_t *d_indices, uint32_t num_tris, const vkg_bvh_build_options *opts,
                                    vkg_bvh **out, void *stream)
{
    return bvh_build(ctx, d_xyz, num_vertices, d_indices, num_tris, opts, grid_wait{}, out, stream);
}

extern "C" vkg_status vkg_diag_build_timeout(vkg_ctx *ctx, const float *d_xyz, uint32_t num_vertices,
                                             const uint32_t *d_indices, uint32_t num_tris, uint64_t limit_ns,
                                             void *stream)
{
    if(!ctx) return VKG_ERR_INVALID_ARGUMENT;
    if(num_tris <= COLLAPSE_PRIMS_PER_BLOCK || limit_ns == 0 || limit_ns > 100000000ull)
        return set_error(ctx, VKG_ERR_INVALID_ARGUMENT, "vkg_diag_build_timeout: need more than %u triangles and 0 < limit_ns <= 1e8",
                         COLLAPSE_PRIMS_PER_BLOCK);
    vkg_bvh *bvh = nullptr;
    const vkg_status s = bvh_build(ctx, d_xyz, num_vertices, d_indices, num_tris, nullptr, grid_wait{limit_ns, 1u}, &bvh, stream);
    vkg_bvh_destroy(ctx, bvh);
    return s;
}

extern "C" vkg_status vkg_bvh_info_get(const vkg_bvh *bvh, vkg_bvh_info *out)
{
    if(!bvh || !out) return VKG_ERR_INVALID_ARGUMENT;
    std::memset(out, 0, sizeof(*out));
    out->num_tris = bvh->num_tris;
    out->num_nodes = bvh->num_nodes;
    out->depth = bvh->depth;
    out->leaf_max = bvh->leaf_max;
    for(int a = 0; a < 3; ++a)
    {
        out->scene_min[a] = bvh->scene_min[a];
        out->scene_max[a] = bvh->scene_max[a];
    }
    out->margin = bvh->margin;
    out->bytes = bvh->bytes;
    out->d_nodes = bvh->d_nodes;
    out->d_tris = bvh->d_tris;
    out->d_morton = bvh->d_morton;
    out->d_sorted = bvh->d_sorted;
    out->build_ms = bvh->build_ms;
    return VKG_OK;
}

// ---- two-level BVH -----------------------------------------------------------------------------
// The top level is the same 8-wide quantised BVH, built by the same core over the instances' world
// boxes (the union of the transformed boxes two levels below a mesh's root, rounded outward); its leaves index
// 128-byte instance records (world <-> object transforms, BLAS, input index, material). Mirrors
// RayBuilder::create_toplevel (RayBuilder.cpp:386-760), which builds the driver TLAS over entries
// carrying a vk_transform_matrix (:518).
extern "C" vkg_status vkg_tlas_build(vkg_ctx *ctx, const vkg_bvh *const *blas, uint32_t num_blas,
                                     const vkg_instance *d_instances, uint32_t num_instances,
                                     const vkg_bvh_build_options *opts, vkg_tlas **out, void *stream_)
{
    if(!ctx) return VKG_ERR_INVALID_ARGUMENT;
    if(!out) return set_error(ctx, VKG_ERR_INVALID_ARGUMENT, "vkg_tlas_build: out is NULL");
    *out = nullptr;
    if(num_instances > 0 && (!d_instances || !blas || num_blas == 0))
        return set_error(ctx, VKG_ERR_INVALID_ARGUMENT, "vkg_tlas_build: NULL instances or BLAS array");
    for(uint32_t b = 0; b < num_blas; ++b)
        if(!blas[b]) return set_error(ctx, VKG_ERR_INVALID_ARGUMENT, "vkg_tlas_build: BLAS %u is NULL", b);
    if(num_instances >= MAX_TRIS)
        return set_error(ctx, VKG_ERR_CAPACITY, "vkg_tlas_build: %u instances exceed the maximum", num_instances);
    const uint32_t leaf_max = (opts && opts->leaf_max) ? opts->leaf_max : 2u;
    if(leaf_max > LEAF_MAX_LIMIT)
        return set_error(ctx, VKG_ERR_INVALID_ARGUMENT, "vkg_tlas_build: leaf_max %u > %u", leaf_max, LEAF_MAX_LIMIT);
    if(vkg_status s = bind_device(ctx); s != VKG_OK) return s;
    cudaStream_t st = static_cast<cudaStream_t>(stream_);
    auto *t = new vkg_tlas();
    t->top.device = ctx->device;
    t->num_instances = num_instances;
    t->num_blas = num_blas;
    t->top.leaf_max = leaf_max;
    std::vector<blas_ref> refs(num_blas);
    std::vector<blas_box> boxes(num_blas);
    for(uint32_t b = 0; b < num_blas; ++b)
    {
        refs[b] = blas_ref{blas[b]->d_nodes, blas[b]->d_tris, blas[b]->num_tris, 0u};
        for(int a = 0; a < 3; ++a)
        {
            boxes[b].lo[a] = blas[b]->scene_min[a];
            boxes[b].hi[a] = blas[b]->scene_max[a];
        }
        boxes[b].num_tris = blas[b]->num_tris;
        t->max_blas_depth = std::max(t->max_blas_depth, blas[b]->depth);
        boxes[b].nodes = blas[b]->d_nodes;
    }
    blas_box *d_bb = nullptr;
    cudaError_t e = cudaSuccess;
    if(num_blas)
    {
        e = dalloc(ctx, &t->d_blas, num_blas, st);
        if(e == cudaSuccess) e = dalloc(ctx, &d_bb, num_blas, st);
        if(e == cudaSuccess)
            e = cudaMemcpyAsync(t->d_blas, refs.data(), num_blas * sizeof(blas_ref), cudaMemcpyHostToDevice, st);
        if(e == cudaSuccess) e = cudaMemcpyAsync(d_bb, boxes.data(), num_blas * sizeof(blas_box), cudaMemcpyHostToDevice, st);
    }
    if(e == cudaSuccess && num_instances)
    {
        e = dalloc(ctx, &t->d_inst, num_instances, st);
        if(e == cudaSuccess) e = dalloc(ctx, &t->d_inst_by_id, num_instances, st);
        if(e == cudaSuccess) e = dalloc(ctx, &t->d_inst_box, 2 * (size_t)num_instances, st);
    }
    if(e != cudaSuccess)
    {
        if(d_bb) cudaFreeAsync(d_bb, st);
        vkg_tlas_destroy(ctx, t);
        return cuda_check(ctx, e, "vkg_tlas_build");
    }
    if(num_instances == 0)
    {
        cudaStreamSynchronize(st);
        if(d_bb) cudaFreeAsync(d_bb, st);
        *out = t;
        return VKG_OK;
    }
    const uint32_t n = num_instances;
    const int T = 256;
    const uint32_t g = (n + T - 1) / T;
    uint32_t err_bits = 0;
    float box_area = 0.f;
    vkg_status s = build_core(
            ctx, &t->top, n, leaf_max, grid_wait{}, st,
            [&](box6 *tbox, uint32_t *scene_enc, uint32_t *err) {
                k_instance_boxes<<<(n + 7) / 8, 256, 0, st>>>(d_instances, n, d_bb, num_blas, tbox, scene_enc, err,
                                                              reinterpret_cast<float *>(scene_enc + 13));
            },
            [&](const uint32_t *sorted, const box6 *lbox, const float *margin) {
                k_instance_records<<<g, T, 0, st>>>(d_instances, sorted, n, num_blas, lbox, margin, t->d_inst,
                                                    t->d_inst_by_id, t->d_inst_box);
            },
            err_bits, box_area);
    if(d_bb) cudaFreeAsync(d_bb, st);
    t->top.num_tris = n;
    const float ex = t->top.scene_max[0] - t->top.scene_min[0], ey = t->top.scene_max[1] - t->top.scene_min[1],
                ez = t->top.scene_max[2] - t->top.scene_min[2], half = ex * ey + ey * ez + ez * ex;
    t->overlap = half > 0.f ? box_area / half : 0.f;
    if(s == VKG_OK && (err_bits & BUILD_ERR_INDEX))
        s = set_error(ctx, VKG_ERR_INVALID_ARGUMENT, "vkg_tlas_build: an instance's BLAS index >= %u", num_blas);
    if(s == VKG_OK && (err_bits & BUILD_ERR_SINGULAR))
        s = set_error(ctx, VKG_ERR_INVALID_ARGUMENT, "vkg_tlas_build: an instance transform is singular");
    if(s == VKG_OK && t->top.depth > TLAS_MAX_DEPTH)
        s = set_error(ctx, VKG_ERR_CAPACITY, "vkg_tlas_build: top-level depth %u exceeds %u", t->top.depth, TLAS_MAX_DEPTH);
    if(s != VKG_OK)
    {
        vkg_tlas_destroy(ctx, t);
        return s;
    }
    t->top.bytes = sizeof(node8) * t->top.num_nodes + (2 * sizeof(inst_rec) + 2 * sizeof(float4)) * (size_t)n;
    *out = t;
    return VKG_OK;
}

extern "C" vkg_status vkg_tlas_info_get(const vkg_tlas *t, vkg_tlas_info *out)
{
    if(!t || !out) return VKG_ERR_INVALID_ARGUMENT;
    std::memset(out, 0, sizeof(*out));
    out->num_instances = t->num_instances;
    out->num_blas = t->num_blas;
    out->num_nodes = t->top.num_nodes;
    out->depth = t->top.depth;
    for(int a = 0; a < 3; ++a)
    {
        out->scene_min[a] = t->top.scene_min[a];
        out->scene_max[a] = t->top.scene_max[a];
    }
    out->d_nodes = t->top.d_nodes;
    out->d_instances = t->d_inst;
    out->d_instances_by_id = t->d_inst_by_id;
    out->build_ms = t->top.build_ms;
    return VKG_OK;
}

// ---- allocation-free build ----------------------------------------------------------------------
// For callers that cannot allocate device memory after start-up (for example an engine that
// sub-allocates everything from one arena it received at initialisation, or code recording work
// that must not synchronise): the build's temporaries live in one file-scope device array of fixed
// size, so the call itself performs no allocation. The caller passes the inputs and the output
// buffers (nodes, triangle records, info words).
namespace vkg
{
namespace
{

constexpr uint32_t NOALLOC_MAX_TRIS = 16384;

struct noalloc_scratch
{
    box6 tbox[NOALLOC_MAX_TRIS], lbox[NOALLOC_MAX_TRIS], ibox[NOALLOC_MAX_TRIS];
    uint32_t keys0[NOALLOC_MAX_TRIS], keys1[NOALLOC_MAX_TRIS], vals0[NOALLOC_MAX_TRIS], vals1[NOALLOC_MAX_TRIS];
    uint32_t counts[sort_count_words(NOALLOC_MAX_TRIS)];
    bvh2_node tree[NOALLOC_MAX_TRIS];
    uint32_t first[NOALLOC_MAX_TRIS];
    uint32_t iparent[NOALLOC_MAX_TRIS], lparent[NOALLOC_MAX_TRIS], visits[NOALLOC_MAX_TRIS];
    uint32_t node_ref[NOALLOC_MAX_TRIS + 8];
    uint32_t morton[NOALLOC_MAX_TRIS];
    uint32_t small[16];
};

// ~2.2 MB, held by every GPU that loads libvkg until the process exits. Host code must not use the
// symbol's host-side name as a device address: the address comes from cudaGetSymbolAddress.
static __device__ __align__(256) unsigned char g_noalloc_scratch[sizeof(noalloc_scratch)];

std::mutex g_noalloc_mutex;
void *g_noalloc_ptr[128] = {};

// per device, on first use, with that device current
vkg_status noalloc_scratch_for_current_device(noalloc_scratch **out)
{
    int dev = -1;
    if(cudaGetDevice(&dev) != cudaSuccess) return VKG_ERR_CUDA;
    if(dev < 0 || dev >= 128) return VKG_ERR_NOT_SUPPORTED;
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if(!g_noalloc_ptr[dev])
    {
        void *p = nullptr;
        cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
        if(e != cudaSuccess || p == nullptr) return VKG_ERR_CUDA;
        g_noalloc_ptr[dev] = p;
    }
    *out = static_cast<noalloc_scratch *>(g_noalloc_ptr[dev]);
    return VKG_OK;
}

// info words: [0] nodes, [1] depth, [2] error flags (1 = index >= num_vertices, 2 = node capacity),
// [3] margin (float bits), [4..6] scene min, [7..9] scene max (float bits)
constexpr uint32_t NOALLOC_FLAG_DEPTH = 4u;

__global__ void k_noalloc_info(const noalloc_scratch *s, uint32_t n, uint32_t *info)
{
    if(threadIdx.x != 0 || blockIdx.x != 0) return;
    for(int k = 0; k < 16; ++k) info[k] = 0u;
    if(n == 0) return;
    info[0] = s->small[8];
    info[1] = s->small[9];
    info[2] = s->small[10] | s->small[6];
    // deeper than the traversal stack supports (the limit vkg_bvh_build enforces)
    if(s->small[9] > (TRAVERSAL_STACK - 1) / 7 + 1) info[2] |= NOALLOC_FLAG_DEPTH;
    info[3] = s->small[12];
    for(int a = 0; a < 3; ++a)
    {
        info[4 + a] = __float_as_uint(fdec(s->small[a]));
        info[7 + a] = __float_as_uint(fdec(s->small[3 + a]));
    }
}

}// namespace
}// namespace vkg

extern "C" vkg_status vkg_bvh_build_noalloc(const float *d_xyz, uint32_t num_vertices, const uint32_t *d_indices,
                                            uint32_t num_tris, uint32_t leaf_max, void *d_nodes,
                                            uint32_t node_capacity, void *d_tris, uint32_t *d_info, void *stream_)
{
    if(num_tris > NOALLOC_MAX_TRIS) return VKG_ERR_CAPACITY;
    if(!d_info) return VKG_ERR_INVALID_ARGUMENT;
    if(leaf_max == 0) leaf_max = 2u;
    if(leaf_max > LEAF_MAX_LIMIT) return VKG_ERR_INVALID_ARGUMENT;
    if(num_tris > 0 && (!d_xyz || !d_indices || num_vertices == 0 || !d_nodes || !d_tris)) return VKG_ERR_INVALID_ARGUMENT;
    if(num_tris > 0 && node_capacity < num_tris) return VKG_ERR_INVALID_ARGUMENT;
    if((reinterpret_cast<uintptr_t>(d_nodes) & 15u) || (reinterpret_cast<uintptr_t>(d_tris) & 15u))
        return VKG_ERR_INVALID_ARGUMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream_);
    noalloc_scratch *s = nullptr;
    if(vkg_status r = noalloc_scratch_for_current_device(&s); r != VKG_OK) return r;
    const uint32_t n = num_tris;
    if(n == 0)
    {
        k_noalloc_info<<<1, 1, 0, st>>>(s, 0, d_info);
        return cudaGetLastError() == cudaSuccess ? VKG_OK : VKG_ERR_CUDA;
    }
    const int T = 256;
    const uint32_t g = (n + T - 1) / T;
    // (the scratch keeps the previous call's contents)
    k_build_init<<<(n + 15 + T - 1) / T, T, 0, st>>>(s->visits, n, s->small);
    k_tri_boxes<<<g, T, 0, st>>>(d_xyz, num_vertices, d_indices, n, s->tbox, s->small, s->small + 6);
    k_morton<<<g, T, 0, st>>>(s->tbox, n, s->small, s->keys0, s->vals0, s->morton);
    uint32_t *kin = s->keys0, *kout = s->keys1, *vin = s->vals0, *vout = s->vals1;
    radix_sort(kin, vin, kout, vout, n, 30, s->counts, st);
    k_gather_leaf_boxes<<<g, T, 0, st>>>(s->tbox, vin, n, s->lbox);
    if(n > 1)
    {
        k_karras<<<(n - 1 + T - 1) / T, T, 0, st>>>(kin, n, s->tree, s->first, s->iparent, s->lparent);
        k_refit<<<g, T, 0, st>>>(s->lparent, s->iparent, s->tree, s->lbox, s->ibox, s->visits, n);
    }
    const uint32_t capacity = std::min<uint32_t>(node_capacity, NOALLOC_MAX_TRIS + 8);
    collapse_args A{s->tree, s->first, s->ibox, s->lbox, n, leaf_max, capacity, s->small, s->node_ref,
                    static_cast<node8 *>(d_nodes), s->small + 8, nullptr, reinterpret_cast<float *>(s->small + 12),
                    grid_wait{}};
    if(launch_collapse(A, 1, st) != cudaSuccess) return VKG_ERR_CUDA;
    k_tri_records<<<g, T, 0, st>>>(d_xyz, num_vertices, d_indices, vin, n, static_cast<tri_rec *>(d_tris));
    k_noalloc_info<<<1, 1, 0, st>>>(s, n, d_info);
    return cudaGetLastError() == cudaSuccess ? VKG_OK : VKG_ERR_CUDA;
}
