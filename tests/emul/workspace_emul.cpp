// workspace_emul.cpp -- the library's memory pools (workspace.cu) against a fake
// CUDA runtime: prints "<name> <value>" per check.
#include <cstdio>
#include <cstdlib>
#include <set>

#include "workspace.cu"

static int g_dev, g_error;
static long g_room = 1000, g_kept[4];  // one memory for all devices; what each pool keeps of it
static cudaMemPool_t pool(int d) { return reinterpret_cast<cudaMemPool_t>(static_cast<size_t>(d + 1)); }
static int dev_of(cudaMemPool_t p) { return (int)reinterpret_cast<size_t>(p) - 1; }

static cudaError_t take(void** p, size_t n)
{
    if ((long)n > g_room) {
        g_error = 1;
        return cudaErrorMemoryAllocation;
    }
    g_room -= (long)n;
    *p = malloc(1);
    return cudaSuccess;
}

extern "C" {
cudaError_t cudaGetDevice(int* d)
{
    *d = g_dev;
    return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps* pr)
{
    if (pr->location.id == 3) return cudaErrorNotSupported;  // a device without pools
    *p = pool(pr->location.id);
    return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t p, size_t)
{
    g_room += g_kept[dev_of(p)];
    g_kept[dev_of(p)] = 0;
    return cudaSuccess;
}
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t q, cudaStream_t)
{
    long& k = g_kept[dev_of(q)];
    if ((long)n <= k) {
        k -= (long)n;
        *p = malloc(1);
        return cudaSuccess;
    }
    return take(p, n);
}
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return take(p, n); }
cudaError_t cudaMalloc(void** p, size_t n) { return take(p, n); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t)
{
    free(p);
    return cudaSuccess;
}
cudaError_t cudaGetLastError(void)
{
    const int e = g_error;
    g_error = 0;
    return e ? cudaErrorMemoryAllocation : cudaSuccess;
}
}

using namespace atmwfs;

int main()
{
    void* p = nullptr;
    auto keep = [&](int dev, long n) {  // a call on `dev` that leaves n bytes in its pool
        g_dev = dev;
        const cudaError_t e = workspace_alloc(&p, (size_t)n, nullptr);
        workspace_free(p, nullptr);
        if (e == cudaSuccess) g_kept[dev] += n;
    };
    keep(0, 300);
    keep(1, 400);
    g_dev = 2;  // released from a device that has no pool
    atmwfs_release_workspaces();
    printf("released_all %d\n", g_kept[0] == 0 && g_kept[1] == 0 && g_room == 1000);
    keep(0, 300);
    keep(1, 400);
    g_dev = 0;
    printf("malloc_makes_room %d\n", device_malloc(&p, 900) == cudaSuccess && p && g_room == 100);
    g_room = 1000;
    keep(1, 600);
    g_dev = 0;
    printf("workspace_makes_room %d\n", workspace_alloc(&p, 700, nullptr) == cudaSuccess && p && g_room == 300);
    g_room = 100;
    printf("failure %d\n", device_malloc(&p, 200) == cudaErrorMemoryAllocation && !p &&
                               workspace_alloc(&p, 200, nullptr) == cudaErrorMemoryAllocation && !p);
    printf("no_error_left %d\n", cudaGetLastError() == cudaSuccess);
    g_dev = 3;
    printf("without_pool %d\n", workspace_alloc(&p, 50, nullptr) == cudaSuccess && p && cudaGetLastError() == cudaSuccess);
    {
        Workspace w(1000, nullptr);
        printf("scope %d\n", w.error() == cudaErrorMemoryAllocation && !w.as<void>());
    }
    return 0;
}
