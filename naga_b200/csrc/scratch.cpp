// Device memory of the set-up primitives' scratch and of the scenes: one
// stream-ordered pool per device that keeps up to kKeep bytes of freed blocks
// (a scene takes ~1.4 KB a node in 3-D; 1 GB is the 100k- to 500k-node
// requests of a serving loop, and 0.6 % of the device).
//
// The device's default pool hands everything back at the next stream
// synchronisation, and the kNN and the weight solves synchronise inside each
// call, so every call mapped its scratch anew: an interpolation of 50,000
// queries that is waited for took 2.5 to 4.2 ms for 2.1 ms of kernels. Blocks
// above kKeep go back to the system at a synchronisation, and all of them
// when an allocation of the library would otherwise fail.
#include <cuda.h>
#include <cuda_runtime.h>

#include <map>
#include <mutex>

#include "scratch.hpp"

namespace naga {

bool current_context_id(unsigned long long* id) {
    using GetCurrent = CUresult (*)(CUcontext*);
    using GetId = CUresult (*)(CUcontext, unsigned long long*);
    static GetCurrent get_current = nullptr;
    static GetId get_id = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", (void**)&get_current, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            get_current = nullptr;
        if (cudaGetDriverEntryPoint("cuCtxGetId", (void**)&get_id, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess)
            get_id = nullptr;
    });
    CUcontext ctx = nullptr;
    if (!get_current || !get_id || get_current(&ctx) != CUDA_SUCCESS || !ctx) return false;
    return get_id(ctx, id) == CUDA_SUCCESS;
}

namespace {

constexpr unsigned long long kKeep = 1ull << 30;

struct Pool {
    unsigned long long context = 0;
    cudaMemPool_t pool = nullptr;  // null: the device has no pools of ours
};
std::mutex g_mu;
std::map<int, Pool> g_pools;

// the current device's pool; null when there is none (the caller then
// allocates from the default pool). A context that was re-created takes a
// new pool: the old one went with its context.
cudaMemPool_t pool_of_device() {
    int dev = 0;
    unsigned long long ctx = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || !current_context_id(&ctx)) {
        cudaGetLastError();
        return nullptr;
    }
    std::lock_guard<std::mutex> lk(g_mu);
    Pool& p = g_pools[dev];
    if (p.context == ctx) return p.pool;
    p.context = ctx;
    p.pool = nullptr;
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.handleTypes = cudaMemHandleTypeNone;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    unsigned long long keep = kKeep;
    if (cudaMemPoolCreate(&p.pool, &props) != cudaSuccess ||
        cudaMemPoolSetAttribute(p.pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) {
        cudaGetLastError();
        p.pool = nullptr;
    }
    return p.pool;
}

}  // namespace

cudaError_t scratch_malloc_bytes(void** p, size_t bytes, cudaStream_t st) {
    *p = nullptr;
    if (cudaMemPool_t pool = pool_of_device()) {
        cudaError_t e = cudaMallocFromPoolAsync(p, bytes, pool, st);
        if (e == cudaErrorMemoryAllocation) {
            cudaGetLastError();
            scratch_trim();
            e = cudaMallocFromPoolAsync(p, bytes, pool, st);
        }
        return e;
    }
    return cudaMallocAsync(p, bytes, st);
}

void scratch_trim() {
    if (cudaMemPool_t pool = pool_of_device())
        if (cudaMemPoolTrimTo(pool, 0) != cudaSuccess) cudaGetLastError();
}

}  // namespace naga
