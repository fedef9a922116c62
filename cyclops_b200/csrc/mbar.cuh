// mbar.cuh -- the exchange between the CTAs of a cluster: 16 bytes stored to a
// peer's shared memory by st.async, counted on the peer's mbarrier.
#pragma once
#include "internal.cuh"

namespace cyc {

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned peer_addr(unsigned addr, int rank) {
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void push16(unsigned dst, unsigned mbar, double a, double b) {
    asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.b64 [%0], {%1, %2}, [%3];" ::"r"(dst),
                 "l"(__double_as_longlong(a)), "l"(__double_as_longlong(b)), "r"(mbar)
                 : "memory");
}
__device__ __forceinline__ void mbar_init(unsigned mbar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mbar) : "memory");
}
__device__ __forceinline__ void mbar_init_fence() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void mbar_expect(unsigned mbar, int bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(unsigned mbar, int phase) {
    unsigned ok;
    asm volatile(
        "{\n.reg .pred p;\n"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok)
        : "r"(mbar), "r"(phase)
        : "memory");
    return ok != 0;
}
// A peer is at most one column's work away (well under a millisecond); a wait
// that outlasts this many clocks (about two seconds) gives up.
constexpr long long kWaitClocks = 4000000000ll;
// waits for the phase; false when the bound ran out
__device__ __forceinline__ bool mbar_wait(unsigned mbar, int phase) {
    if (mbar_try(mbar, phase)) return true;
    const long long t0 = clock64();
    while (!mbar_try(mbar, phase))
        if (clock64() - t0 > kWaitClocks) return false;
    return true;
}

}  // namespace cyc
