// vkg_bvh_destroy / vkg_tlas_destroy against a recording stand-in for the CUDA runtime with two devices: the
// memory of a tree goes back only after its own device has been waited for, whichever device is current
// and with or without a context, and the device that was current stays so.
#include "../../vierkant_gb300/csrc/internal.hpp"

#include <cstdio>

static int g_current = 0, g_waits[2], g_frees, g_early;
static int g_device; // the tree's

extern "C" {
cudaError_t cudaGetDevice(int *d) { return *d = g_current, cudaSuccess; }
cudaError_t cudaSetDevice(int d) { return g_current = d, cudaSuccess; }
cudaError_t cudaDeviceSynchronize(void) { return ++g_waits[g_current], cudaSuccess; }
cudaError_t cudaFree(void *p)
{
    if(!p) return cudaSuccess;
    ++g_frees;
    g_early += g_waits[g_device] == 0;
    return cudaSuccess;
}
}
vkg_status vkg::bind_device(vkg_ctx *ctx) { return g_current = ctx->device, VKG_OK; }

static char g_memory[8];
template<class T>
static T *mem(int i)
{
    return reinterpret_cast<T *>(g_memory + i);
}

int main()
{
    int bad = 0;
    for(int tree = 0; tree < 2; ++tree)
        for(int current = 0; current < 2; ++current)
            for(int with_ctx = 0; with_ctx < 2; ++with_ctx)
                for(int two_level = 0; two_level < 2; ++two_level)
                {
                    g_device = tree;
                    g_current = current;
                    g_waits[0] = g_waits[1] = g_frees = g_early = 0;
                    vkg_ctx ctx;
                    ctx.device = tree;
                    vkg_ctx *c = with_ctx ? &ctx : nullptr;
                    if(two_level)
                    {
                        auto *t = new vkg_tlas();
                        t->top.device = tree;
                        t->top.d_nodes = mem<vkg::node8>(0);
                        t->top.d_morton = mem<uint32_t>(1);
                        t->top.d_sorted = mem<uint32_t>(2);
                        t->d_inst = mem<vkg::inst_rec>(3);
                        t->d_inst_by_id = mem<vkg::inst_rec>(4);
                        t->d_inst_box = mem<float4>(5);
                        t->d_blas = mem<vkg::blas_ref>(6);
                        vkg_tlas_destroy(c, t);
                    }
                    else
                    {
                        auto *b = new vkg_bvh();
                        b->device = tree;
                        b->d_nodes = mem<vkg::node8>(0);
                        b->d_tris = mem<vkg::tri_rec>(1);
                        b->d_morton = mem<uint32_t>(2);
                        b->d_sorted = mem<uint32_t>(3);
                        vkg_bvh_destroy(c, b);
                    }
                    // (a call with a context leaves the context's device current, as every call does)
                    const bool ok = g_frees == (two_level ? 7 : 4) && g_early == 0 && g_current == (with_ctx ? tree : current);
                    if(!ok)
                        std::printf("tree on %d, current %d, context %d, two levels %d: %d freed, %d before the wait, current %d\n",
                                    tree, current, with_ctx, two_level, g_frees, g_early, g_current);
                    bad += !ok;
                }
    return bad != 0;
}
