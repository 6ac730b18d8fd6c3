// Host stand-in for eimp_b200/csrc/async_copy.cuh under the warp emulator: an
// mbarrier is a phase count and its pending arrivals; a bulk copy is done at
// once and arrives on its barrier in place of the expected bytes.
#pragma once
#include "emu.h"
namespace eimp {
constexpr int MBAR_POLLS = 1 << 28;   // polls are far shorter here than on the device
struct EmuMbar { std::atomic<int> pending; std::atomic<short> phase; short count; };
static_assert(sizeof(EmuMbar) == 8, "stored in a barrier's 64 bits");
inline EmuMbar *emu_mbar(uint64_t *b) { return reinterpret_cast<EmuMbar *>(b); }
inline void mbar_init(uint64_t *b, int n) {
    emu_mbar(b)->pending = n;
    emu_mbar(b)->phase = 0;
    emu_mbar(b)->count = (short)n;
}
inline void mbar_init_fence() {}
inline void mbar_arrive(uint64_t *b) {
    if (emu_mbar(b)->pending.fetch_sub(1) == 1) {
        emu_mbar(b)->pending += emu_mbar(b)->count;
        emu_mbar(b)->phase++;
    }
}
inline void mbar_expect(uint64_t *, unsigned) {}
inline bool mbar_try(uint64_t *b, unsigned parity) {
    sched_yield();
    return (unsigned)(emu_mbar(b)->phase.load() & 1) != (parity & 1u);
}
inline bool mbar_wait(uint64_t *b, unsigned parity) {
    while ((unsigned)(emu_mbar(b)->phase.load() & 1) == (parity & 1u)) sched_yield();
    return true;
}
inline void bulk_load(void *dst, const void *src, unsigned bytes, uint64_t *b) {
    if ((bytes | (uintptr_t)dst | (uintptr_t)src) & 15) { fprintf(stderr, "bulk copy off 16 bytes\n"); abort(); }
    memcpy(dst, src, bytes);
    mbar_arrive(b);
}
inline void emu_copy(void *dst, const void *src, size_t n) {
    if (((uintptr_t)dst | (uintptr_t)src) & (n - 1)) { fprintf(stderr, "asynchronous copy off %zu bytes\n", n); abort(); }
    memcpy(dst, src, n);
}
inline void copy_async16(void *dst, const void *src) { emu_copy(dst, src, 16); }
inline void copy_async8(void *dst, const void *src) { emu_copy(dst, src, 8); }
inline void copy_async_commit() {}
template <int N> inline void copy_async_wait() {}
inline void block_barrier(int) { emu_block->arrive_and_wait(); }
inline void pair_barrier(int k, int threads) {   // among warps of the same block
    static EmuBarrier bars[4];
    bars[k].n = threads;
    bars[k].arrive_and_wait();
}
}  // namespace eimp
