// umma_core.cuh -- tcgen05 building blocks of the surrogate's products: the
// shared-memory and instruction descriptors, tensor-memory allocation and
// reads, and the bounded waits.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace atmwfs {
namespace umma {

constexpr int kM = 128;      // pixels per tile (MMA M, one TMEM lane each)
constexpr int kThreads = 256;
constexpr uint64_t kWaitNs = 1000000000ull;

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ uint64_t now_ns()
{
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Shared-memory matrix descriptor, no swizzle, K-major: core matrices of 8
// rows x 16 bytes; `lbo` = byte distance of core matrices along K, `sbo` =
// along M/N (8-row groups); bits 46-47 = 1 (descriptor version of sm_100).
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo)
{
    uint64_t d = 0;
    d |= (uint64_t)((addr >> 4) & 0x3FFF);
    d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
    d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
    d |= (uint64_t)1 << 46;
    return d;  // base offset 0, layout type 0 (no swizzle)
}

// Instruction descriptor of kind::f16: D FP32, A and B BF16, both K-major,
// N = n, M = 128.
__host__ __device__ constexpr uint32_t instr_desc(int n)
{
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kM >> 4) << 24);
}

__device__ __forceinline__ void mbar_init(uint64_t* bar)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(bar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_addr(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// 16 consecutive TMEM columns of this warp's 32 lanes: register j = column c0 + j.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&r)[16])
{
    uint32_t u[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
        : "=r"(u[0]), "=r"(u[1]), "=r"(u[2]), "=r"(u[3]), "=r"(u[4]), "=r"(u[5]), "=r"(u[6]), "=r"(u[7]),
          "=r"(u[8]), "=r"(u[9]), "=r"(u[10]), "=r"(u[11]), "=r"(u[12]), "=r"(u[13]), "=r"(u[14]), "=r"(u[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 16; j++) r[j] = __uint_as_float(u[j]);
}

// Byte offset of element (row, k) in a K-major no-swizzle tile with kc = K/8
// core matrices per 8-row group (LBO = 128 B, SBO = kc * 128 B).
__device__ __forceinline__ uint32_t kmajor_off(int row, int k, int kc)
{
    return (uint32_t)((row >> 3) * kc * 128 + (k >> 3) * 128 + (row & 7) * 16 + (k & 7) * 2);
}

// Tensor memory of the CTA: `cols` columns (a power of two >= 32), allocated
// and freed by warp 0; the base is read after the next barrier.
__device__ __forceinline__ void tmem_alloc(uint32_t* base, uint32_t cols, int warp)
{
    if (warp != 0) return;
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(base)), "r"(cols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(uint32_t base, uint32_t cols, int warp)
{
    __syncthreads();
    if (warp != 0) return;
    fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(base), "r"(cols) : "memory");
}

// The CTA's shared-memory stores become visible to the tensor core (which
// reads through the async proxy) and the CTA meets.
__device__ __forceinline__ void publish_smem()
{
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    fence_before();
    __syncthreads();
    fence_after();
}

// The CTA has read a tile's results: its operands and accumulators are free.
__device__ __forceinline__ void retire_tile()
{
    fence_before();
    __syncthreads();
    fence_after();
}

// D (+)= A B^T for one K step of 16 (one thread issues).
__device__ __forceinline__ void mma_bf16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool accumulate)
{
    const uint32_t acc = accumulate ? 1u : 0u;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(acc)
        : "memory");
}

__device__ __forceinline__ void mma_commit(uint64_t* bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar))
                 : "memory");
}

// Every thread waits for the committed products, at most 1 s; the CTA agrees
// on the outcome.  false: the wait ran out (the status bit is set).
__device__ __forceinline__ bool mma_wait(uint64_t* bar, uint32_t parity, unsigned* status)
{
    const uint64_t t0 = now_ns();
    int timed_out = 0;
    while (!mbar_try_wait(bar, parity)) {
        if (now_ns() - t0 > kWaitNs) {
            timed_out = 1;
            break;
        }
    }
    if (__syncthreads_or(timed_out)) {
        if (threadIdx.x == 0 && status) atomicOr(status, 1u);
        return false;
    }
    fence_after();
    return true;
}

}  // namespace umma
}  // namespace atmwfs
