// Thread-block-cluster primitives shared by the sweep kernels (sm_103a).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "brr_device.cuh"

namespace brr {

// ---- thread-block-cluster primitives (distributed shared memory)
__device__ __forceinline__ unsigned cl_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

// Address of the same shared-memory location in CTA `rank` of the cluster.
__device__ __forceinline__ unsigned cl_map(unsigned addr, unsigned rank)
{
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}

// 16-byte store into a CTA's shared memory that completes as 16 transaction
// bytes on that CTA's mbarrier `rbar`.
__device__ __forceinline__ void cl_push16(unsigned raddr, unsigned long long w0, unsigned long long w1, unsigned rbar)
{
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(raddr),
                 "l"(w0), "l"(w1), "r"(rbar)
                 : "memory");
}

__device__ __forceinline__ void cl_bar_init(uint64_t *m)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(cl_addr(m)) : "memory");
}

// The receiver's own arrival of a round: one arrival plus the bytes it expects.
__device__ __forceinline__ void cl_expect(uint64_t *m, unsigned bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(cl_addr(m)), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool cl_test(uint64_t *m, unsigned parity)
{
    unsigned ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.test_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok)
                 : "r"(cl_addr(m)), "r"(parity)
                 : "memory");
    return ok != 0;
}

// Waits for phase `parity` of m at most timeout_ns; false on timeout.
__device__ __forceinline__ bool cl_wait(uint64_t *m, unsigned parity, uint64_t timeout_ns)
{
    if (cl_test(m, parity))
        return true;
    const uint64_t t0 = global_timer_ns();
    unsigned spins = 0;
    while (!cl_test(m, parity)) {
        if ((++spins & 63u) == 0 && global_timer_ns() - t0 > timeout_ns)
            return false;
    }
    return true;
}

// All threads of all CTAs of the cluster (release / acquire at cluster scope).
// Used once after the mbarriers are initialised and once before the CTAs
// exit; every wait between the two is bounded, so every CTA reaches both.
__device__ __forceinline__ void cl_sync_all()
{
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

__device__ __forceinline__ unsigned cl_rank()
{
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

}  // namespace brr
