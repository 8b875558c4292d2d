// Destruction of the BVHs. Their memory is stream-ordered, and cudaFree does not wait for work that still reads
// such memory (as it does for cudaMalloc's): a query may be under way on any stream, so the tree's device is
// waited for first. The tree knows its device: a call without a context may come with another one current.
#include "internal.hpp"

namespace
{

void release(vkg_ctx *ctx, int device, std::initializer_list<void *> memory)
{
    if(ctx) vkg::bind_device(ctx);
    int current = device;
    cudaGetDevice(&current);
    if(current != device) cudaSetDevice(device);
    cudaDeviceSynchronize();
    for(void *p: memory) cudaFree(p);
    if(current != device) cudaSetDevice(current);
}

}// namespace

extern "C" {

vkg_status vkg_bvh_destroy(vkg_ctx *ctx, vkg_bvh *bvh)
{
    if(!bvh) return VKG_OK;
    release(ctx, bvh->device, {bvh->d_nodes, bvh->d_tris, bvh->d_morton, bvh->d_sorted});
    delete bvh;
    return VKG_OK;
}

vkg_status vkg_tlas_destroy(vkg_ctx *ctx, vkg_tlas *t)
{
    if(!t) return VKG_OK;
    release(ctx, t->top.device,
            {t->top.d_nodes, t->top.d_morton, t->top.d_sorted, t->d_inst, t->d_inst_by_id, t->d_inst_box, t->d_blas});
    delete t;
    return VKG_OK;
}

}// extern "C"
