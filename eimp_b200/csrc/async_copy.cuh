// Asynchronous copies from global to shared memory: bulk copies that complete
// on an mbarrier (cp.async.bulk), with bounded waits, and per-thread copies in
// groups (cp.async).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace eimp {

// Polls after which a wait gives up.  A poll (mbarrier.try_wait) suspends the
// thread for a hardware-chosen time of at most a few microseconds, so the limit
// is seconds -- far beyond any copy -- and a kernel whose barrier is never
// completed still ends.
constexpr int MBAR_POLLS = 1 << 20;

__device__ __forceinline__ unsigned smem_addr(const void *p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t *bar, int arrivals) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(arrivals) : "memory");
}
// makes the initialised barriers visible to the copy engine
__device__ __forceinline__ void mbar_init_fence() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("{ .reg .b64 t; mbarrier.arrive.shared::cta.b64 t, [%0]; }" ::"r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ void mbar_expect(uint64_t *bar, unsigned bytes) {
    asm volatile("{ .reg .b64 t; mbarrier.arrive.expect_tx.shared::cta.b64 t, [%0], %1; }" ::"r"(smem_addr(bar)),
                 "r"(bytes)
                 : "memory");
}
// one poll for the phase with the given parity: true when it is complete
__device__ __forceinline__ bool mbar_try(uint64_t *bar, unsigned parity) {
    unsigned done;
    asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                 : "=r"(done)
                 : "r"(smem_addr(bar)), "r"(parity)
                 : "memory");
    return done != 0;
}
// waits for it; false when it gave up
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, unsigned parity) {
    for (int i = 0; i < MBAR_POLLS; i++)
        if (mbar_try(bar, parity)) return true;
    return false;
}
// bytes (a multiple of 16) from global src to shared dst, both 16-byte aligned
__device__ __forceinline__ void bulk_load(void *dst, const void *src, unsigned bytes, uint64_t *bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_addr(dst)),
                 "l"(src), "r"(bytes), "r"(smem_addr(bar))
                 : "memory");
}


// 16 or 8 bytes by the calling thread, both addresses aligned to the size
__device__ __forceinline__ void copy_async16(void *dst, const void *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_async8(void *dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
// closes the calling thread's group of copies
__device__ __forceinline__ void copy_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// waits until at most N of the calling thread's groups are in flight
template <int N> __device__ __forceinline__ void copy_async_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// a barrier of 'threads' threads of the CTA, reached from any place in the code
__device__ __forceinline__ void block_barrier(int threads) { asm volatile("bar.sync 1, %0;" ::"r"(threads) : "memory"); }
// further ones, by number
__device__ __forceinline__ void pair_barrier(int k, int threads) {
    asm volatile("bar.sync %0, %1;" ::"r"(1 + k), "r"(threads) : "memory");
}

}  // namespace eimp
