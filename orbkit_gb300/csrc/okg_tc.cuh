// Blackwell building blocks shared by the tensor-core kernels: mbarriers with bounded
// waits, bulk copies, tcgen05 commits, fences and tensor-memory loads.
#pragma once
#include <stdint.h>

namespace okg {
namespace mx {

constexpr long long WAIT_LIMIT = 1ll << 24;

__device__ __forceinline__ uint32_t smem_u32(const void* p)
{
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mma_commit(uint32_t bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}

__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}

// Bounded wait: returns false if the phase does not complete within `limit` polls.
__device__ __forceinline__ bool mbar_try_for(uint32_t bar, uint32_t parity, long long limit)
{
    for (long long it = 0; it < limit; ++it)
        if (mbar_try(bar, parity)) return true;
    return false;
}

// The same, also raising the status word if the phase does not
// complete within `limit` polls (WAIT_LIMIT unless the plan sets another).
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, int* status, long long limit)
{
    if (mbar_try_for(bar, parity, limit)) return true;
    atomicExch(status, 1);
    return false;
}

// Wait for the completion of the CTA's own asynchronous work (a bulk copy or
// MMAs) before it leaves: bounded by WAIT_LIMIT whatever the plan's limit, since
// such work always completes; false if even that expires.
__device__ __forceinline__ bool mbar_drain(uint32_t bar, uint32_t parity)
{
    return mbar_try_for(bar, parity, WAIT_LIMIT);
}

// Whether any thread of the CTA raised the abort flag, the same answer for every
// lane of the calling warp (all 32 lanes must call it): decisions that lead to
// warp-collective instructions (tcgen05.ld, shuffles) stay uniform.
__device__ __forceinline__ bool warp_aborted(const int* flag)
{
    return __any_sync(0xffffffffu, *(const volatile int*)flag != 0);
}

__device__ __forceinline__ void mbar_arrive(uint32_t bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}

// One bulk copy global -> shared (16-byte aligned addresses, size a multiple of
// 16) completing on an mbarrier that expects `bytes` transaction bytes.
__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

__device__ __forceinline__ void fence_proxy_async()
{
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr));
}

}  // namespace mx
}  // namespace okg
