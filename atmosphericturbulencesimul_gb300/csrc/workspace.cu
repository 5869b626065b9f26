// workspace.cu -- the library's memory pool (workspace.cuh).
#include <map>
#include <mutex>

#include "workspace.cuh"

namespace atmwfs {

namespace {
std::mutex g_mu;
std::map<int, cudaMemPool_t> g_pools;  // one per device; null where none could be made

cudaMemPool_t pool_of(int dev, bool create)
{
    std::lock_guard<std::mutex> lk(g_mu);
    const auto it = g_pools.find(dev);
    if (it != g_pools.end()) return it->second;
    if (!create) return nullptr;
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
}  // namespace

cudaError_t workspace_alloc(void** p, size_t bytes, cudaStream_t st)
{
    *p = nullptr;
    int dev = 0;
    const cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const cudaMemPool_t pool = pool_of(dev, true);
    return pool ? cudaMallocFromPoolAsync(p, bytes, pool, st) : cudaMallocAsync(p, bytes, st);
}

void workspace_free(void* p, cudaStream_t st)
{
    if (p) cudaFreeAsync(p, st);
}

void workspace_release()
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return;
    if (const cudaMemPool_t pool = pool_of(dev, false)) cudaMemPoolTrimTo(pool, 0);
}

}  // namespace atmwfs
