// workspace.cu -- the library's memory pool (workspace.cuh).
#include <map>
#include <mutex>

#include "atmwfs.h"
#include "workspace.cuh"

namespace atmwfs {

namespace {
std::mutex g_mu;
std::map<int, cudaMemPool_t> g_pools;  // one per device; null where none could be made

cudaMemPool_t pool_of(int dev)
{
    std::lock_guard<std::mutex> lk(g_mu);
    const auto it = g_pools.find(dev);
    if (it != g_pools.end()) return it->second;
    cudaMemPoolProps pr = {};
    pr.allocType = cudaMemAllocationTypePinned;
    pr.location.type = cudaMemLocationTypeDevice;
    pr.location.id = dev;
    cudaMemPool_t p = nullptr;
    if (cudaMemPoolCreate(&p, &pr) == cudaSuccess) {
        unsigned long long keep = kWorkspaceKeep;
        cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep);
    } else {
        cudaGetLastError();
        p = nullptr;
    }
    g_pools[dev] = p;
    return p;
}

// get(), and once more with what the pools keep given back where that could help.
template <typename F>
cudaError_t with_room(void** p, F get)
{
    *p = nullptr;
    cudaError_t e = get();
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        workspace_release();
        e = get();
    }
    if (e != cudaSuccess) {
        cudaGetLastError();  // reported here, not by a later launch
        *p = nullptr;
    }
    return e;
}
}  // namespace

cudaError_t workspace_alloc(void** p, size_t bytes, cudaStream_t st)
{
    *p = nullptr;
    int dev = 0;
    const cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const cudaMemPool_t pool = pool_of(dev);
    return with_room(p, [&] { return pool ? cudaMallocFromPoolAsync(p, bytes, pool, st) : cudaMallocAsync(p, bytes, st); });
}

cudaError_t device_malloc(void** p, size_t bytes)
{
    return with_room(p, [&] { return cudaMalloc(p, bytes); });
}

void workspace_free(void* p, cudaStream_t st)
{
    if (p) cudaFreeAsync(p, st);
}

void workspace_release()
{
    std::lock_guard<std::mutex> lk(g_mu);
    for (const auto& q : g_pools)
        if (q.second) cudaMemPoolTrimTo(q.second, 0);
}

}  // namespace atmwfs

extern "C" void atmwfs_release_workspaces(void) { atmwfs::workspace_release(); }
