// Shared-memory loads, mbarriers with bounded waits and bulk copies of the quantised products (qgemv.cu, gemm_quant_tc.cu).
#pragma once
#include <stdint.h>

namespace juno {

__device__ __forceinline__ uint4 lds128(uint32_t a) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a));
    return v;
}
__device__ __forceinline__ uint32_t lds32(uint32_t a) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
    return v;
}
__device__ __forceinline__ uint32_t lds16(uint32_t a) {
    uint32_t v;
    asm volatile("{\n.reg .u16 h;\nld.shared.u16 h, [%1];\ncvt.u32.u16 %0, h;\n}\n" : "=r"(v) : "r"(a));
    return v;
}

// ── mbarrier / bulk-copy primitives ──────────────────────────────────────────────────────
__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, unsigned count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
// One attempt.  ns == 0: a plain test.  Otherwise the hardware may park the warp for up to about `ns` nanoseconds when
// the phase is not complete yet (fewer issue slots than polling, but it wakes late when the hint is long).
__device__ __forceinline__ bool mbar_test(uint32_t bar, unsigned parity, unsigned ns) {
    unsigned ok;
    if (ns == 0)
        asm volatile(
            "{\n.reg .pred p;\n"
            "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n"
            "selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok)
            : "r"(bar), "r"(parity)
            : "memory");
    else
        asm volatile(
            "{\n.reg .pred p;\n"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n"
            "selp.u32 %0, 1, 0, p;\n}\n"
            : "=r"(ok)
            : "r"(bar), "r"(parity), "r"(ns)
            : "memory");
    return ok != 0;
}
// Weight tiles are read once per step: they are requested with the evict-first policy, so that the gigabytes streamed
// through the L2 do not push out what every kernel start needs again (activations, norm weights, instructions).
__device__ __forceinline__ uint64_t l2_evict_first_policy() {
    uint64_t pol;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(pol));
    return pol;
}
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void *src, unsigned bytes, uint32_t bar, uint64_t pol) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1], %2, [%3], %4;" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar), "l"(pol)
                 : "memory");
}
// A wait on a weight tile gives up after this many SM cycles (about a fifth of a second); after the first give-up
// of a warp its later waits are short, so that the kernel still drains the copies it has in flight and returns.
constexpr long long kQWaitLimitClk = 400000000ll, kQWaitLimitAfterFail = 2000000ll;
__device__ __forceinline__ void mbar_wait_bounded(uint32_t bar, unsigned parity, unsigned ns, unsigned *err, bool &failed) {
    if (mbar_test(bar, parity, 0)) return;
    const long long t0 = clock64(), limit = failed ? kQWaitLimitAfterFail : kQWaitLimitClk;
    while (!mbar_test(bar, parity, ns)) {
        if (clock64() - t0 > limit) {
            if (!failed && (threadIdx.x & 31) == 0) *reinterpret_cast<volatile unsigned *>(err) = 1u | ((threadIdx.x >> 5) << 8) | (blockIdx.x << 16);
            failed = true;
            return;
        }
    }
}

}  // namespace juno
