// Shared-memory barriers, bounded waits on them, and bulk copies that report to them (sm_100a).
#pragma once

#include "common.cuh"

namespace sessd {

// About a tenth of a second. Waits are microseconds: whoever waits for another role of its block is behind the wait for the
// preceding kernel (which may run for any time) where that role is.
constexpr long long WAIT_LIMIT_CYCLES = 200000000LL;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// More bytes for the current phase to wait for (a thread whose own arrival for the phase is still to come says so).
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.expect_tx.relaxed.cta.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// As mbar_try_wait, but the hardware may park the thread for up to `ns` nanoseconds while the phase is incomplete,
// so a waiting warp does not take issue slots from the warps that feed the pipeline.
__device__ __forceinline__ bool mbar_try_wait_parked(uint32_t bar, uint32_t parity, uint32_t ns) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity), "r"(ns)
        : "memory");
    return ok != 0;
}
// Bounded wait: false when the phase did not complete within the clock limit or the CTA is aborting.
// The polling loop is kept to a handful of instructions (abort flag and clock are looked at every 32
// polls). RELAXED waits (roles with slack: weight and index prefetch) also sleep between polls. The MMA
// issuers use the plain limit, every other role one and a half times that: when something upstream is
// missing, the wait closest to the cause is the one that gets reported.
template <bool RELAXED = false, bool ISSUER = false>
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag, int where = 0) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    const long long limit = ISSUER ? WAIT_LIMIT_CYCLES : WAIT_LIMIT_CYCLES + WAIT_LIMIT_CYCLES / 2;
    for (;;) {
#pragma unroll 1
        for (int i = 0; i < 32; ++i) {
            if (RELAXED) __nanosleep(200);
            if (mbar_try_wait_parked(bar, parity, 1000u)) return true;
        }
        if (*abort_flag) return false;
        if (clock64() - t0 > limit) {
            if (*abort_flag == 0) abort_flag[1] = where;   // abort_where follows abort_flag in SharedCtl
            *abort_flag = 1;
            return false;
        }
    }
}

__device__ __forceinline__ void bulk_load(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar)
                 : "memory");
}

}  // namespace sessd
