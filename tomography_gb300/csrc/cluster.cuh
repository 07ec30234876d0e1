// Thread-block clusters: barriers, addresses in the other blocks' shared memory, and
// the exchange of halo rows.
#pragma once
#include <cuda_runtime.h>

namespace tomo {

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned cluster_blocks() {
    unsigned r;
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned remote_addr(unsigned local, unsigned rank) {
    unsigned r;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
    return r;
}
// A halo row travels as one bulk copy between the shared memories: it counts its
// bytes on an mbarrier of the receiving block, whose reader waits for them.
// Neighbours need no other synchronisation.  (A cluster barrier per step waits for the
// slowest block of all and costs a fence for the block's global stores: 5.6 us a step on
// 400^2 where this took 4.1.  Stores of 16 bytes, one count each, took 4.3.)
__device__ __forceinline__ void mbar_init(unsigned bar) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arm(unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try(unsigned bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ void proxy_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void copy_row(unsigned dst, unsigned src, unsigned bytes, unsigned bar) {
    asm volatile("cp.async.bulk.shared::cluster.shared::cta.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "r"(src), "r"(bytes), "r"(bar)
                 : "memory");
}
// A word of another block's shared memory.  That block has to be still running.
__device__ __forceinline__ void remote_store(unsigned addr, int v) {
    asm volatile("st.shared::cluster.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory");
}
__device__ __forceinline__ int remote_load(unsigned addr) {
    int v;
    asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}

// Waits for a halo row; false when it did not come within about two seconds, which no
// correct run meets, or when `lost` says that the cluster has given up.
constexpr long long kHaloClocks = 4000000000ll;
__device__ __forceinline__ bool mbar_wait(unsigned bar, unsigned parity, const volatile int* lost) {
    if (mbar_try(bar, parity)) return true;
    const long long start = clock64();
    while (clock64() - start < kHaloClocks && !(lost && *lost))
        if (mbar_try(bar, parity)) return true;
    return false;
}

// A place in the block's dynamic shared memory.  Pointers kept in memory lose
// their address space (and cost generic loads), so tables are kept as offsets.
template <typename T>
__device__ __forceinline__ T* shared_at(size_t offset) {
    extern __shared__ __align__(16) unsigned char smem[];
    return reinterpret_cast<T*>(smem + offset);
}

}  // namespace tomo
