// Host stand-in for eimp_b200/csrc/async_copy.cuh under the warp emulator: an
// mbarrier is a phase count and its pending arrivals; a bulk copy is done at
// once and arrives on its barrier in place of the expected bytes.
#pragma once
#include "emu.h"
namespace eimp {
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
inline bool mbar_wait(uint64_t *b, unsigned parity) {
    while ((unsigned)(emu_mbar(b)->phase.load() & 1) == (parity & 1u)) sched_yield();
    return true;
}
inline void bulk_load(void *dst, const void *src, unsigned bytes, uint64_t *b) {
    if ((bytes | (uintptr_t)dst | (uintptr_t)src) & 15) { fprintf(stderr, "bulk copy off 16 bytes\n"); abort(); }
    memcpy(dst, src, bytes);
    mbar_arrive(b);
}
}  // namespace eimp
