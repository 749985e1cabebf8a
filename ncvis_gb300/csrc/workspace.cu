// The library's memory pool (common.cuh): one per device and context.
#include <cuda.h>
#include <cuda_runtime.h>

#include <map>
#include <mutex>
#include <string>
#include <utility>

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

std::mutex g_mu;
// By device and context id; ids are not used again, so the entry of a context that
// was destroyed, whose pool went with it, is never met.  Never destroyed: an engine
// may outlive the library's static objects.
using Pools = std::map<std::pair<int, unsigned long long>, cudaMemPool_t>;
Pools &g_pools = *new Pools;

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
    unsigned long long id = current_context_id();
    if (id == 0) {
        // A thread that has made no call which needs a context yet.
        NCVIS_CUDA(cudaFree(nullptr));
        id = current_context_id();
        require(id != 0, "workspace pool: no current context", kCudaError);
    }
    std::lock_guard<std::mutex> lock(g_mu);
    cudaMemPool_t &known = g_pools[{dev, id}];
    if (!known) {
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
        known = pool;
    }
    return known;
}

void trim_workspace_pool(int dev) {
    int current = 0;
    if (cudaGetDevice(&current) != cudaSuccess) return;
    if (dev != current && cudaSetDevice(dev) != cudaSuccess) return;
    try {
        std::lock_guard<std::mutex> lock(g_mu);
        const auto known = g_pools.find({dev, current_context_id()});
        if (known != g_pools.end() && known->second) cudaMemPoolTrimTo(known->second, 0);
    } catch (const Error &) {  // no context any more: nothing is kept either
    }
    if (dev != current) cudaSetDevice(current);
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
