// Internal host-side state shared by the libvkg translation units (not part of the C ABI).
#pragma once

#include "../../include/vkg.h"
#include "../../include/vkg_diag.h"
#include "vkg_common.cuh"

#include <cuda_runtime.h>

#include <cstdarg>
#include <cstdio>
#include <initializer_list>
#include <string>

namespace vkg
{
// Scratch of the binnings (traverse.cu): the context's, grown on demand, whose uses on different streams are ordered
// by an event; or a view of memory whose owner's calls follow one another anyway (bin_view, no event).
// keys: bin | rank in its tile << 16 per element; perm: position -> element (its first half holds the
// 16-bit bins before that); tile_counts: elements per (tile, bin); bin_totals: first positions of runs of
// 32 bins and of the bins within them, the counters of the binning; done: recorded after the last use,
// waited for by the next
struct bin_scratch
{
    uint32_t *keys = nullptr;
    uint32_t *perm = nullptr;
    uint32_t *tile_counts = nullptr;
    uint32_t *bin_totals = nullptr;
    size_t cap = 0;
    uint32_t tiles_cap = 0;
    cudaEvent_t done = nullptr;
    bool view = false;
    void release_buffers() // cudaFree waits for the device, so nothing in flight still uses them
    {
        for(uint32_t *p: {keys, perm, tile_counts, bin_totals}) cudaFree(p);
        keys = perm = tile_counts = bin_totals = nullptr;
        cap = 0;
        tiles_cap = 0;
    }
    void release()
    {
        release_buffers();
        if(done) cudaEventDestroy(done);
        done = nullptr;
    }
};
}// namespace vkg

struct vkg_ctx
{
    int device = 0;
    int num_sms = 0;
    std::string last_error;
    // Stream-ordered memory of the builds and of per-call scratch (ctx_alloc). Unused memory up to
    // POOL_KEEP stays with the pool when a stream is waited for, where the device's default pool would
    // hand it back and map it again at the next call (a build paid 0.3 ms for that, a 720p denoise and
    // post-FX 0.36 ms); destroyed with the context.
    cudaMemPool_t pool = nullptr;
    // device counters: [0] node visits, [1] triangle tests, [2] error flags (bit0 stack overflow)
    unsigned long long *d_counters = nullptr;
    // ray index counter of the persistent traversal kernels
    uint32_t *d_work = nullptr;
    // host-variant staging (grown on demand)
    void *d_stage_rays = nullptr;
    void *d_stage_hits = nullptr;
    size_t stage_rays_bytes = 0, stage_hits_bytes = 0;
    // the host variant's copy / trace pipeline (created on first use): streams [0], [1] trace
    // alternate chunks, [2] uploads, [3] downloads; events: [0] fork, [1..4] joins, [5] a chunk's
    // upload done, [6] a chunk's trace done
    cudaStream_t pipe[4] = {nullptr, nullptr, nullptr, nullptr};
    cudaEvent_t pipe_ev[7] = {nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr};
    vkg::bin_scratch bins; // of the ray queries and the path tracer
};

struct vkg_bvh
{
    int device = 0; // where its memory lies
    uint32_t num_tris = 0, num_nodes = 0, depth = 0, leaf_max = 4;
    float scene_min[3] = {0, 0, 0}, scene_max[3] = {0, 0, 0}, margin = 0.f;
    vkg::node8 *d_nodes = nullptr;
    vkg::tri_rec *d_tris = nullptr;
    uint32_t *d_morton = nullptr; // input order
    uint32_t *d_sorted = nullptr; // sorted order -> triangle id
    size_t bytes = 0;
    float build_ms = 0.f;
};

namespace vkg
{
// instance record of a two-level BVH (128 B): world->object and object->world 3x4 row-major
// transforms, the BLAS the instance refers to, its input index and material
struct alignas(16) inst_rec
{
    float w2o[12];
    float o2w[12];
    uint32_t blas, instance, material, pad0;
    uint32_t pad1[4];
};
static_assert(sizeof(inst_rec) == 128, "inst_rec layout");

// top-level traversal stack; the build rejects top levels deeper than it supports
constexpr uint32_t TLAS_STACK = 64;
constexpr uint32_t TLAS_MAX_DEPTH = (TLAS_STACK - 1) / 7 + 1;

// a bottom-level BVH as the top level sees it
struct alignas(16) blas_ref
{
    const node8 *nodes;
    const tri_rec *tris;
    uint32_t num_tris, pad;
};
}// namespace vkg

struct vkg_tlas
{
    vkg_bvh top;                       // 8-wide BVH over the instances' world boxes (no triangle records)
    vkg::inst_rec *d_inst = nullptr;   // instance records in sorted (leaf) order
    vkg::inst_rec *d_inst_by_id = nullptr; // the same records in input order
    float4 *d_inst_box = nullptr;      // world boxes in leaf order, grown by the margin: {lo xyz, hi x}, {hi yz, -, -}
    vkg::blas_ref *d_blas = nullptr;
    uint32_t num_instances = 0, num_blas = 0;
    uint32_t max_blas_depth = 0; // depth of the deepest mesh BVH
    float overlap = 0.f; // instance boxes that a random line through the scene crosses, on average
};

namespace vkg
{
constexpr uint64_t POOL_KEEP = 512ull << 20;
// memory from the context's pool, ordered on `st`; freed with cudaFreeAsync, or with cudaFree once no
// work that uses it is in flight
inline cudaError_t ctx_alloc(vkg_ctx *ctx, void **p, size_t bytes, cudaStream_t st)
{
    return cudaMallocFromPoolAsync(p, bytes, ctx->pool, st);
}

// record an error message on ctx and return `status`
vkg_status set_error(vkg_ctx *ctx, vkg_status status, const char *fmt, ...);
// map a CUDA error to VKG_ERR_CUDA with location info; VKG_OK if err == cudaSuccess
vkg_status cuda_check(vkg_ctx *ctx, cudaError_t err, const char *what);
// ensure the context's device is current on this thread
vkg_status bind_device(vkg_ctx *ctx);

// traversal stack capacity (entries) of the traversal kernels; the build rejects deeper BVHs
constexpr uint32_t TRAVERSAL_STACK = 128;

// Ray binning (traverse.cu): the order in which to trace the rays d_rays[0, n) -- or [0, *d_n) when
// d_n is a device-side count <= n -- so that neighbouring threads follow similar paths through bvh:
// perm[position] = ray, valid when *reordered_out (a device word) is non-zero; otherwise the rays
// are to be traced as given. Returns nullptr (trace as given) for VKG_RAY_KEEP_ORDER, batches below
// min_rays, a stream being captured, or scratch that cannot be allocated. The scratch is the
// context's (ctx->bins); calls on different streams are ordered by an event recorded by bins_done().
const uint32_t *bin_rays(vkg_ctx *ctx, const vkg_bvh *bvh, const vkg_ray *d_rays, uint32_t n, const uint32_t *d_n,
                         uint32_t flags, uint32_t min_rays, cudaStream_t st, const uint32_t **reordered_out);
// Batches from which binning pays. The binning itself takes 40-90 us; a closest-hit traversal of incoherent
// rays gains more than that from 2^19 rays on (600,000: 441 -> 414 us, 784,000: 531 -> 494 us), an any-hit
// traversal, which ends at the first hit, from about 1.5 million (bounce rays, 600,000: 164 -> 184 us, 784,000:
// 209 -> 218 us, 1,200,000: 351 either way, 1,800,000: 551 -> 534 us; camera rays, 1,048,576: 176 -> 203 us; rays all
// over the scene's box gain earlier, 700,000: 331 -> 325 us, 1,048,576: 472 -> 439 us).
constexpr uint32_t BIN_MIN_CLOSEST = 1u << 19, BIN_MIN_ANY = 3u << 19;
// the same for points (the first three floats of records of `stride` floats) over a 32^3 grid of the box
// lo, 1 / scale: neighbouring positions of the order are neighbouring in space; `bins` is the caller's scratch.
// Fewer than min_points points, by n or by *d_n, keep their order
const uint32_t *bin_points(vkg_ctx *ctx, bin_scratch &bins, const float *d_points, uint32_t stride, uint32_t n,
                           const uint32_t *d_n, const float lo[3], const float scale[3], uint32_t min_points,
                           cudaStream_t st, const uint32_t **reordered_out);
// after the launch that reads the order: the scratch may be reused once the stream reaches here
inline void bins_done(const bin_scratch &bins, cudaStream_t st)
{
    if(!bins.view) cudaEventRecord(bins.done, st);
}
// scratch for n elements in `bytes` bytes at mem (256-byte aligned); of no use to bin_points if they are too few
bin_scratch bin_view(const vkg_ctx *ctx, uint32_t n, void *mem, size_t bytes);
}// namespace vkg

#define VKG_TRY_CUDA(ctx, expr)                                                                                      \
    do                                                                                                               \
    {                                                                                                                \
        vkg_status s_ = vkg::cuda_check((ctx), (expr), #expr);                                                       \
        if(s_ != VKG_OK) return s_;                                                                                  \
    } while(0)
