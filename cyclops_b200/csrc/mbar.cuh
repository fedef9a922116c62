// mbar.cuh -- the exchange between the CTAs of a cluster: 16 bytes stored to a
// peer's shared memory by st.async, counted on the peer's mbarrier.
#pragma once
#include <cstdio>
#include <cstdlib>

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
// waits for the phase; false when `clocks` ran out (0: without a look)
__device__ __forceinline__ bool mbar_wait(unsigned mbar, int phase, long long clocks) {
    if (clocks <= 0) return false;
    if (mbar_try(mbar, phase)) return true;
    const long long t0 = clock64();
    while (!mbar_try(mbar, phase))
        if (clock64() - t0 > clocks) return false;
    return true;
}
// before the CTAs of a cluster that lost one another leave: stores of 16 bytes
// that nobody waited for land within a few microseconds; about 50 pass here
__device__ __forceinline__ void stores_land() {
    const long long t0 = clock64();
    while (clock64() - t0 < 100000) {}
}

// How long a CTA waits for its peers.  A peer is at most one pass over its rows
// away, and in the worst case (one stratum, one thread) that pass is a chain of
// dependent loads and exponentials, 1,000 to 1,500 clocks a row; so two seconds
// and 4,096 clocks a row of the CTA with the most.  CYC_WAIT_CLOCKS="clocks[,rank]"
// sets the bound, and takes CTA `rank` of every cluster for lost at its first
// wait (how the tests reach this path).
struct WaitLimit {
    long long clocks;
    int lost;
    __device__ __forceinline__ long long of(int rank) const { return rank == lost ? 0 : clocks; }
};
inline WaitLimit wait_limit(long long rows) {
    WaitLimit w{4000000000ll + 4096 * rows, -1};
    if (const char* e = std::getenv("CYC_WAIT_CLOCKS")) std::sscanf(e, "%lld,%d", &w.clocks, &w.lost);
    return w;
}

}  // namespace cyc
