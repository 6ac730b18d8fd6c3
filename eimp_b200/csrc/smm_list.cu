// Set-maximal matches without mismatches (setmaxerrors = 0, the reference's
// default) for B200 (sm_100a).
//
//  smm_list_kernel -- TargetImp::calcSMMatches / processHistorySubTree
//                     (TargetImp.cpp:74-246, 346-435), one warp per target
//                     haplotype.
//
// The reference keeps a tree of PBWT intervals; stored in pre-order, a site
// turns it into [new root] ++ {0-extensions} ++ {1-extensions}, each part in
// the old order, and then replaces a node whose only child has its interval
// by that child.  Without mismatches two things follow:
//  * two nodes of which neither descends from the other hold disjoint sets of
//    haplotypes: they were separated at a site the target misses, one by each
//    allele.  So equal intervals mean ancestor and descendant, which are next
//    to each other in pre-order when no node lies between them, and a node's
//    second child would make its first child's interval smaller than its own.
//    The merge is therefore "drop an entry whose successor has its interval";
//    parents and sides need not be stored;
//  * a node's depth is the current site minus the site it started at, so a
//    node never has to be rewritten for its depth.
// The tree is a list of (start, interval), and a site the target does not
// miss only filters it: one interval end pair mapped per node, in place.
//
// The list is kept in reverse pre-order (deepest branch first, the root last):
// a dropped entry then repeats the interval of the entry before it, so one
// pass over 32 entries at a time knows what to drop, and the new root is
// appended.
//
// What bounds it: the chain from one site to the next (list entry -> two PBWT
// words -> ballots -> list entry).  The PBWT rows come through shared memory
// where they fit (16-bit interval ends: at most 65,536 haplotypes): a
// producer warp streams groups of consecutive rows into a ring with bulk
// copies, every warp of the CTA reads them at shared-memory latency, and each
// row crosses L2 once per CTA.  Wider rows are read in place.
//
// Measured on a B200 against the general kernel (smm_compact_kernel): 1,000
// haplotypes x 5,000 sites of a 10,000-haplotype panel 19.2 -> 4.6 ms; 128 x
// 3,000 of 20,000 haplotypes 11.7 -> 2.7 ms; 64 x 2,000 of 200,000 haplotypes
// (rows in place) 12.9 -> 4.6 ms.
#include <climits>

#include "async_copy.cuh"
#include "common.cuh"
#include "kernels.h"

namespace eimp {

constexpr int SL_CAP = 512;         // list entries per warp in shared memory
constexpr int SL_POOL = SMM_NODES_RETRY;   // entries of a global pool, the most a list may hold
constexpr int SL_RETRY = -2;        // nmatch mark: redone by the general kernel's retry launch
constexpr int SL_WARPS = 23;        // target haplotypes per CTA, at most (what shared memory holds)
constexpr int SL_STAGES = 4;        // groups of rows in the ring

// an interval [l, r] of PBWT positions in one word
template <bool WIDE> struct SlIv;
template <> struct SlIv<false> {
    typedef uint32_t T;
    static __device__ __forceinline__ T pack(int l, int r) { return (uint32_t)l | ((uint32_t)r << 16); }
    static __device__ __forceinline__ int l(T v) { return (int)(v & 0xffffu); }
    static __device__ __forceinline__ int r(T v) { return (int)(v >> 16); }
};
template <> struct SlIv<true> {
    typedef unsigned long long T;
    static __device__ __forceinline__ T pack(int l, int r) { return (T)(uint32_t)l | ((T)(uint32_t)r << 32); }
    static __device__ __forceinline__ int l(T v) { return (int)(uint32_t)v; }
    static __device__ __forceinline__ int r(T v) { return (int)(v >> 32); }
};

template <bool WIDE, int CAP> struct SlList {
    typename SlIv<WIDE>::T iv[2][CAP];
    int st[2][CAP];
};

__device__ __forceinline__ unsigned sl_lt() { return (1u << (threadIdx.x & 31)) - 1u; }

// zeros of a compressed PBWT row at the positions before i, and up to i
__device__ __forceinline__ int sl_zeros_before(const uint2 *row, int i) {
    const uint2 p = row[i >> 5];
    return (int)p.y - __popc(~p.x & (~0u << (i & 31)));
}
__device__ __forceinline__ int sl_zeros_upto(const uint2 *row, int i) {
    const uint2 p = row[i >> 5];
    return (int)p.y - __popc(~p.x & ~((2u << (i & 31)) - 1u));
}

// The rows as one warp reads them: in place, or from the CTA's ring of
// SL_STAGES groups of 'group' consecutive rows.
struct SlRows {
    const uint8_t *compr;
    size_t rowbytes;
    int M, group;           // group 0: rows are read in place
    const uint8_t *ring;
    size_t stage_bytes;
    uint64_t *full, *empty;
    int stage;
    unsigned parity;
    const uint8_t *cur;     // the next row
    int left;               // rows left in the current group (staged)
    int site;               // rows done
    bool ok;                // no wait gave up

    __device__ __forceinline__ void open() {
        stage = 0; parity = 0u; left = 0; site = 0; ok = true;
        cur = compr;
    }
    // the row of site 'site'
    __device__ __forceinline__ const uint2 *next() {
        if (group && left == 0) {
            ok = ok && mbar_wait(&full[stage], parity);
            // the copy starts at the 16-byte boundary at or before the group
            cur = ring + (size_t)stage * stage_bytes + (((size_t)site * rowbytes) & 15);
            left = min(group, M - site);
        }
        const uint2 *row = reinterpret_cast<const uint2 *>(cur);
        cur += rowbytes;
        return row;
    }
    // all lanes are done with the row last taken
    __device__ __forceinline__ void done() {
        __syncwarp();
        site++;
        if (group && --left == 0) {
            if ((threadIdx.x & 31) == 0) mbar_arrive(&empty[stage]);
            if (++stage == SL_STAGES) { stage = 0; parity ^= 1u; }
        }
    }
};

struct SlState {
    int n;       // entries of the list, the root last
    int cur;     // which of the two buffers holds it
    int nres;    // matches written
    int tdst;    // start of the deepest entries (their depth: site - tdst)
    uint32_t err;
};

// the matches [nres, nres + cnt) were written in list order: turn them into pre-order
__device__ __forceinline__ void sl_reverse(int4 *out, int nres, int cnt) {
    __syncwarp();
    for (int j = threadIdx.x & 31; j < cnt / 2; j += 32) {
        const int4 a = out[nres + j], b = out[nres + cnt - 1 - j];
        out[nres + j] = b;
        out[nres + cnt - 1 - j] = a;
    }
    __syncwarp();
}

// The sites [m, M] of one haplotype on a list of CAP entries.  Returns M + 1
// when it is done or failed (s.err), or -- with can_switch -- the first site
// that could outgrow the list, before touching it.
template <bool WIDE, int CAP>
__device__ __forceinline__ int sl_sites(SlList<WIDE, CAP> &L, SlState &s, SlRows &rows, int m, bool can_switch, int K,
                                        int nwords, const uint8_t *__restrict__ g, const uint32_t *__restrict__ hw,
                                        int4 *__restrict__ out, int cap) {
    typedef SlIv<WIDE> IV;
    typedef typename IV::T T;
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned lt = sl_lt();
    const int M = rows.M;
    const T NONE = IV::pack(1, 0);   // no interval
    const int m0 = m;
    unsigned missw = 0u, currw = 0u;
    int nextg = 0;
    unsigned nexth = 0u;
    {   // the 32 sites m lies in
        const int b = m & ~31;
        const int gv = b + lane < M ? g[b + lane] : 0;
        missw = __ballot_sync(FULL, gv == 3);
        currw = b < M ? hw[b >> 5] : 0u;
        nextg = b + 32 + lane < M ? g[b + 32 + lane] : 0;
        nexth = b + 32 < M ? hw[(b >> 5) + 1] : 0u;
    }
    for (; m < M; m++) {
        if (can_switch && 2 * s.n + 1 > CAP) return m;
        if ((m & 31) == 0 && m != m0) {
            missw = __ballot_sync(FULL, nextg == 3);
            currw = nexth;
            nextg = m + 32 + lane < M ? g[m + 32 + lane] : 0;
            nexth = m + 32 < M ? hw[(m >> 5) + 1] : 0u;
        }
        const bool missing = (missw >> (m & 31)) & 1u;
        const bool curr = (currw >> (m & 31)) & 1u;
        const uint2 *row = rows.next();
        if (!rows.ok) { s.err |= EIMP_ERR_WAIT; return M + 1; }
        const int c0 = (int)row[nwords - 1].y;   // the row's zeros
        const bool hastd = s.tdst < m;           // an entry deeper than the root exists
        T *iv = L.iv[s.cur];
        int *st = L.st[s.cur];
        int newcount = 0, kept = 0, alln = 1;
        bool anydeep = false;
        int minst = INT_MAX;
        if (!missing) {
            T carry = NONE;
            for (int base = 0; base < s.n; base += 32) {
                const int i = base + lane;
                bool alive = false, deep = false;
                T v = NONE;
                int start = 0, l = 0, r = -1;
                if (i < s.n) {
                    const T x = iv[i];
                    start = st[i];
                    l = IV::l(x); r = IV::r(x);
                    const int zl = sl_zeros_before(row, l), zr = sl_zeros_upto(row, r);
                    const int nl = curr ? c0 + l - zl : zl, nr = curr ? c0 + r - zr : zr - 1;
                    alive = nl <= nr;
                    v = IV::pack(nl, nr);
                    deep = hastd && start == s.tdst;
                }
                const unsigned ba = __ballot_sync(FULL, alive), bd = __ballot_sync(FULL, deep && !alive);
                const unsigned below = ba & lt;
                T p = __shfl_sync(FULL, v, below ? 31 - __clz((int)below) : 0);
                if (!below) p = carry;
                const bool keep = alive && p != v;
                const unsigned bk = __ballot_sync(FULL, keep);
                if (deep && !alive) {
                    const int pos = s.nres + newcount + __popc(bd & lt);
                    if (pos < cap) out[pos] = make_int4(start, m, l, r);
                    else s.err |= EIMP_ERR_MATCH_OVERFLOW;
                }
                anydeep |= deep && alive;
                if (alive) minst = min(minst, start);
                if (keep) {   // at or before the entry just read: in place
                    const int q = kept + __popc(bk & lt);
                    iv[q] = v;
                    st[q] = start;
                }
                if (ba) carry = __shfl_sync(FULL, v, 31 - __clz((int)ba));
                kept += __popc(bk);
                alln += __popc(ba);
                newcount += __popc(bd);
            }
        } else {
            // both extensions: the 1-extensions, then the 0-extensions, into
            // the other buffer
            T *oiv = L.iv[s.cur ^ 1];
            int *ost = L.st[s.cur ^ 1];
            for (int ext = 1; ext >= 0; ext--) {
                T carry = NONE;
                for (int base = 0; base < s.n; base += 32) {
                    const int i = base + lane;
                    bool alive = false, dead = false, deep = false;
                    T v = NONE;
                    int start = 0, l = 0, r = -1;
                    if (i < s.n) {
                        const T x = iv[i];
                        start = st[i];
                        l = IV::l(x); r = IV::r(x);
                        const int zl = sl_zeros_before(row, l), zr = sl_zeros_upto(row, r);
                        const bool a0 = zl <= zr - 1, a1 = l - zl <= r - zr;
                        alive = ext ? a1 : a0;
                        v = ext ? IV::pack(c0 + l - zl, c0 + r - zr) : IV::pack(zl, zr - 1);
                        deep = hastd && start == s.tdst;
                        dead = ext && deep && !a0 && !a1;
                    }
                    const unsigned ba = __ballot_sync(FULL, alive), bd = __ballot_sync(FULL, dead);
                    const unsigned below = ba & lt;
                    T p = __shfl_sync(FULL, v, below ? 31 - __clz((int)below) : 0);
                    if (!below) p = carry;
                    const bool keep = alive && p != v;
                    const unsigned bk = __ballot_sync(FULL, keep);
                    if (dead) {
                        const int pos = s.nres + newcount + __popc(bd & lt);
                        if (pos < cap) out[pos] = make_int4(start, m, l, r);
                        else s.err |= EIMP_ERR_MATCH_OVERFLOW;
                    }
                    anydeep |= deep && alive;
                    if (alive) minst = min(minst, start);
                    if (keep) {
                        const int q = kept + __popc(bk & lt);
                        if (q < CAP) { oiv[q] = v; ost[q] = start; }
                    }
                    if (ba) carry = __shfl_sync(FULL, v, 31 - __clz((int)ba));
                    kept += __popc(bk);
                    alln += __popc(ba);
                    newcount += __popc(bd);
                }
            }
            s.cur ^= 1;
            iv = oiv;
            st = ost;
        }
        // the entries before any merge are what the general kernel's pool
        // must hold: refused at the same count
        if (alln > CAP) { s.err |= EIMP_ERR_NODE_OVERFLOW; rows.done(); return M + 1; }
        if (lane == 0) { iv[kept] = IV::pack(0, K - 1); st[kept] = m + 1; }
        s.n = kept + 1;
        if (!__any_sync(FULL, anydeep)) {
            // the deepest entries end here: set-maximal (TargetImp.cpp:132-136)
            if (newcount && s.nres + newcount <= cap) {
                if (newcount > 1) sl_reverse(out, s.nres, newcount);
                s.nres += newcount;
            }
            for (int o = 16; o; o >>= 1) minst = min(minst, __shfl_xor_sync(FULL, minst, o));
            s.tdst = min(minst, m + 1);
        }
        rows.done();
    }
    // TargetImp.cpp:144: the erase pass, the deepest entries report
    if (s.tdst < M) {
        const T *iv = L.iv[s.cur];
        const int *st = L.st[s.cur];
        int newcount = 0;
        for (int base = 0; base < s.n; base += 32) {
            const int i = base + lane;
            const bool deep = i < s.n && st[i] == s.tdst;
            const unsigned bd = __ballot_sync(FULL, deep);
            if (deep) {
                const int pos = s.nres + newcount + __popc(bd & lt);
                if (pos < cap) out[pos] = make_int4(s.tdst, M, IV::l(iv[i]), IV::r(iv[i]));
                else s.err |= EIMP_ERR_MATCH_OVERFLOW;
            }
            newcount += __popc(bd);
        }
        if (s.nres + newcount <= cap) {
            if (newcount > 1) sl_reverse(out, s.nres, newcount);
            s.nres += newcount;
        }
    }
    return M + 1;
}

template <bool WIDE>
__global__ void __launch_bounds__((SL_WARPS + 1) * 32) smm_list_kernel(
    const uint32_t *__restrict__ compr, int M, int K, const uint64_t *__restrict__ phased, int wM,
    const uint8_t *__restrict__ gt, int nhaps, const int32_t *__restrict__ hapmap, int4 *__restrict__ matches, int cap,
    int *__restrict__ nmatch, uint32_t *__restrict__ status, int warps, int group, unsigned stage_bytes,
    SlList<WIDE, SL_POOL> *__restrict__ gpool, int gpool_slots, int *__restrict__ gpool_next) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int h0 = blockIdx.x * warps;
    const int live = min(warps, nhaps - h0);   // haplotypes of this CTA
    const int nwords = (K + 31) / 32;
    uint64_t *full = reinterpret_cast<uint64_t *>(smem_raw), *empty = full + SL_STAGES;
    uint8_t *ring = smem_raw + 2 * SL_STAGES * sizeof(uint64_t);
    SlList<WIDE, SL_CAP> *lists =
        reinterpret_cast<SlList<WIDE, SL_CAP> *>(ring + (group ? (size_t)SL_STAGES * stage_bytes : 0));
    SlRows rows;
    rows.compr = reinterpret_cast<const uint8_t *>(compr);
    rows.rowbytes = (size_t)nwords * 8;
    rows.M = M; rows.group = group;
    rows.ring = ring; rows.stage_bytes = stage_bytes;
    rows.full = full; rows.empty = empty;
    if (group) {
        if (threadIdx.x == 0) {
            for (int i = 0; i < SL_STAGES; i++) { mbar_init(&full[i], 1); mbar_init(&empty[i], live); }
            mbar_init_fence();
        }
        __syncthreads();
        if (wid == warps) {   // the producer: one thread copies group after group
            if (lane == 0) {
                const int ngroups = (M + group - 1) / group;
                int stage = 0, gi = 0;
                unsigned parity = 1u;   // a fresh barrier's previous phase counts as done
                bool ok = true;
                for (; gi < ngroups; gi++) {
                    if (!mbar_wait(&empty[stage], parity)) { ok = false; break; }
                    const size_t a = (size_t)gi * group * rows.rowbytes;
                    const size_t b = min((size_t)(gi + 1) * group, (size_t)M) * rows.rowbytes;
                    const size_t a16 = a & ~(size_t)15, b16 = (b + 15) & ~(size_t)15;
                    mbar_expect(&full[stage], (unsigned)(b16 - a16));
                    bulk_load(ring + (size_t)stage * stage_bytes, rows.compr + a16, (unsigned)(b16 - a16), &full[stage]);
                    if (++stage == SL_STAGES) { stage = 0; parity ^= 1u; }
                }
                if (!ok) atomicOr(status, (uint32_t)EIMP_ERR_WAIT);
                // the copies in flight end before the CTA does
                for (int j = max(0, gi - SL_STAGES); j < gi; j++)
                    mbar_wait(&full[j % SL_STAGES], (unsigned)(j / SL_STAGES) & 1u);
            }
            return;
        }
    }
    if (wid >= live) return;
    const int hap = hapmap ? hapmap[h0 + wid] : h0 + wid;   // the haplotypes that exist (PBWTImputer.cpp:130)
    const uint8_t *g = gt + (size_t)(hap >> 1) * M;
    const uint32_t *hw = reinterpret_cast<const uint32_t *>(phased + (size_t)hap * wM);
    int4 *out = matches + (size_t)hap * cap;
    const unsigned FULL = 0xffffffffu;
    rows.open();
    // missingness > 50 %: no matches (TargetImp.cpp:79-80)
    int nmiss = 0;
#pragma unroll 4
    for (int m = lane; m < M; m += 32) nmiss += g[m] == 3;
    for (int o = 16; o; o >>= 1) nmiss += __shfl_xor_sync(FULL, nmiss, o);
    SlState s;
    s.n = 1; s.cur = 0; s.nres = 0; s.tdst = 0; s.err = 0u;
    if (nmiss <= M / 2) {
        SlList<WIDE, SL_CAP> &L = lists[wid];
        if (lane == 0) { L.iv[0][0] = SlIv<WIDE>::pack(0, K - 1); L.st[0][0] = 0; }
        __syncwarp();
        const int m = sl_sites<WIDE, SL_CAP>(L, s, rows, 0, gpool != nullptr, K, nwords, g, hw, out, cap);
        if (m <= M) {   // the list could outgrow shared memory: on in a global pool
            int slot = 0;
            if (lane == 0) slot = atomicAdd(gpool_next, 1);
            slot = __shfl_sync(FULL, slot, 0);
            if (slot < gpool_slots) {
                SlList<WIDE, SL_POOL> &G = gpool[slot];
                for (int i = lane; i < s.n; i += 32) { G.iv[0][i] = L.iv[s.cur][i]; G.st[0][i] = L.st[s.cur][i]; }
                s.cur = 0;
                __syncwarp();
                sl_sites<WIDE, SL_POOL>(G, s, rows, m, false, K, nwords, g, hw, out, cap);
            } else {
                sl_sites<WIDE, SL_CAP>(L, s, rows, m, false, K, nwords, g, hw, out, cap);
            }
        }
    }
    // a haplotype that ended early still releases the rows the others wait for
    while (group && rows.ok && rows.site < M) {
        rows.next();
        if (rows.ok) rows.done();
        else s.err |= EIMP_ERR_WAIT;
    }
    for (int o = 16; o; o >>= 1) s.err |= __shfl_xor_sync(FULL, s.err, o);
    if (lane) return;
    if (!s.err) { nmatch[hap] = s.nres; return; }
    if (s.err == EIMP_ERR_NODE_OVERFLOW) { nmatch[hap] = SL_RETRY; return; }
    nmatch[hap] = -1;
    atomicOr(status, s.err);
}

// ---------------------------------------------------------------------------
// launcher
// ---------------------------------------------------------------------------
size_t smm_list_slot_bytes(int K) { return K <= 65536 ? sizeof(SlList<false, SL_POOL>) : sizeof(SlList<true, SL_POOL>); }

template <bool WIDE>
static cudaError_t smm_list_launch(const uint32_t *compr, int M, int K, const uint64_t *phased, int wM,
                                   const uint8_t *gt, int nhaps, const int32_t *hapmap, int4 *matches, int cap,
                                   int *nmatch, uint32_t *status, void *gpool, int gpool_slots, int *gpool_next,
                                   cudaStream_t st) {
    int dev = 0, nsm = 0, lim = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&lim, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e != cudaSuccess) return e;
    // narrow intervals (at most 65,536 haplotypes, rows up to 16 KB): the rows
    // go through the ring, about 8 KB a group, and the haplotypes are spread
    // over the SMs with as many to a CTA as one even number of waves needs.
    // Wide: rows in place, nothing shared in a CTA.
    const size_t rowbytes = (size_t)((K + 31) / 32) * 8, list = sizeof(SlList<WIDE, SL_CAP>);
    int group = 0;
    size_t stage = 0;
    if (!WIDE) {
        group = (int)(8192 / rowbytes);
        group = group < 1 ? 1 : group > 16 ? 16 : group;
        stage = (group * rowbytes + 30) & ~(size_t)15;   // a copy starts up to 15 bytes before its rows
    }
    const size_t head = 2 * SL_STAGES * sizeof(uint64_t) + SL_STAGES * stage;
    int most = (int)(((size_t)lim - head) / list);
    most = most > SL_WARPS ? SL_WARPS : most;
    if (WIDE && most > 4) most = 4;
    int warps = (nhaps + nsm - 1) / nsm;
    if (warps > most) {
        const int waves = WIDE ? 1 : (nhaps + most * nsm - 1) / (most * nsm);
        warps = WIDE ? most : (nhaps + waves * nsm - 1) / (waves * nsm);
    }
    const size_t sm = head + (size_t)warps * list;
    if ((e = ensure_dynamic_smem((const void *)smm_list_kernel<WIDE>, sm)) != cudaSuccess) return e;
    smm_list_kernel<WIDE><<<(nhaps + warps - 1) / warps, (warps + (group ? 1 : 0)) * 32, sm, st>>>(
        compr, M, K, phased, wM, gt, nhaps, hapmap, matches, cap, nmatch, status, warps, group, (unsigned)stage,
        static_cast<SlList<WIDE, SL_POOL> *>(gpool), gpool_slots, gpool_next);
    return cudaGetLastError();
}

cudaError_t launch_smm_list(const uint32_t *compr, int M, int K, const uint64_t *phased, int wM, const uint8_t *gt,
                            int nhaps, const int32_t *hapmap, int4 *matches, int cap, int *nmatch, uint32_t *status,
                            void *gpool, int gpool_slots, int *gpool_next, cudaStream_t st) {
    if (K <= 65536)
        return smm_list_launch<false>(compr, M, K, phased, wM, gt, nhaps, hapmap, matches, cap, nmatch, status, gpool,
                                      gpool_slots, gpool_next, st);
    return smm_list_launch<true>(compr, M, K, phased, wM, gt, nhaps, hapmap, matches, cap, nmatch, status, gpool,
                                 gpool_slots, gpool_next, st);
}

}  // namespace eimp
