// The library's memory pool (common.cuh): one per device and context.
#include <cuda.h>
#include <cuda_runtime.h>

#include <mutex>
#include <string>

#include "common.cuh"

namespace ncvis_gpu {

namespace {

using CtxGetCurrentFn = CUresult (*)(CUcontext *);
using CtxGetIdFn = CUresult (*)(CUcontext, unsigned long long *);

template <class Fn>
Fn driver_entry(const char *name) {
    void *p = nullptr;
    cudaDriverEntryPointQueryResult q;
    NCVIS_CUDA(cudaGetDriverEntryPointByVersion(name, &p, 12000, cudaEnableDefault, &q));
    require(q == cudaDriverEntryPointSuccess && p != nullptr,
            std::string("driver entry point ") + name + " is unavailable", kCudaError);
    return (Fn)p;
}

constexpr int kMaxDevices = 128;
struct Pool {
    unsigned long long ctx_id = 0;
    cudaMemPool_t pool = nullptr;
};
std::mutex g_mu;
Pool g_pools[kMaxDevices];

}  // namespace

unsigned long long current_context_id() {
    static const CtxGetCurrentFn get_current = driver_entry<CtxGetCurrentFn>("cuCtxGetCurrent");
    static const CtxGetIdFn get_id = driver_entry<CtxGetIdFn>("cuCtxGetId");
    CUcontext ctx = nullptr;
    require(get_current(&ctx) == CUDA_SUCCESS, "cuCtxGetCurrent failed", kCudaError);
    if (!ctx) return 0;
    unsigned long long id = 0;
    require(get_id(ctx, &id) == CUDA_SUCCESS, "cuCtxGetId failed", kCudaError);
    return id;
}

cudaMemPool_t workspace_pool() {
    int dev = 0;
    NCVIS_CUDA(cudaGetDevice(&dev));
    require(dev >= 0 && dev < kMaxDevices, "device index out of range");
    std::lock_guard<std::mutex> lock(g_mu);
    const unsigned long long id = current_context_id();
    Pool &e = g_pools[dev];
    if (id == 0 || e.ctx_id != id || !e.pool) {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t pool = nullptr;
        NCVIS_CUDA(cudaMemPoolCreate(&pool, &props));
        uint64_t keeps = kPoolKeeps;
        const cudaError_t set =
            cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keeps);
        if (set != cudaSuccess) {
            cudaMemPoolDestroy(pool);
            NCVIS_CUDA(set);
        }
        e.pool = pool;  // a pool of an earlier context went with it
        e.ctx_id = current_context_id();
    }
    return e.pool;
}

void trim_workspace_pool() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return;
    std::lock_guard<std::mutex> lock(g_mu);
    const Pool &e = g_pools[dev];
    if (!e.pool) return;
    try {
        if (e.ctx_id == current_context_id()) cudaMemPoolTrimTo(e.pool, 0);
    } catch (const Error &) {  // no context any more: nothing is kept either
    }
}

void *pool_alloc(size_t bytes, cudaStream_t s) {
    const cudaMemPool_t pool = workspace_pool();
    void *p = nullptr;
    const size_t n = bytes > 0 ? bytes : 1;
    cudaError_t r = cudaMallocFromPoolAsync(&p, n, pool, s);
    if (r == cudaErrorMemoryAllocation) {
        // What the pool keeps in pieces of other sizes may be what is missing.
        cudaGetLastError();
        NCVIS_CUDA(cudaStreamSynchronize(s));
        NCVIS_CUDA(cudaMemPoolTrimTo(pool, 0));
        r = cudaMallocFromPoolAsync(&p, n, pool, s);
    }
    NCVIS_CUDA(r);
    return p;
}

}  // namespace ncvis_gpu
