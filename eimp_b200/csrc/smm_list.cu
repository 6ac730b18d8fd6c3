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
// What bounds it: for many haplotypes the instructions of the lookups (an entry
// is two PBWT words and 27 instructions a site, sl_run), for few the chain from
// one site to the next.  The PBWT rows come through shared memory where they
// fit (16-bit interval ends: at most 65,536 haplotypes): a producer warp
// streams groups of consecutive rows into a ring with bulk copies, every warp
// of the CTA reads them at shared-memory latency, and each row crosses L2 once
// per CTA.  Wider rows are read in place.
//
// Few haplotypes are searched in several chunks of sites each (grid.y).  A
// chunk starts with the root alone and takes over the matches that start
// behind its first site: the entries that start later are the same whether or
// not deeper ones are listed before them (those only hide equal intervals,
// which end when they do), and the first of them to report is known when the
// entry of the chunk's first site ends.  Past its last site a chunk adds no
// roots and goes on until its list is empty, so that together the chunks map
// no entry twice.
//
// Measured on a B200: the general kernel (smm_compact_kernel), one site at a
// time in one chunk, and now.  1,000 haplotypes x 5,000 sites of a
// 10,000-haplotype panel 19.2, 4.6, 1.91 ms; 128 x 3,000 of 20,000 haplotypes
// 11.7, 2.7, 0.39 ms; 64 x 2,000 of 200,000 haplotypes (rows in place) 12.9, 4.6,
// 0.40 ms; 400 x 2,000 of 5,000 haplotypes, the last two, 1.34, 0.32 ms.
#include <climits>

#include "async_copy.cuh"
#include "common.cuh"
#include "kernels.h"

namespace eimp {

constexpr int SL_CAP = 512;         // list entries per warp in shared memory
constexpr int SL_POOL = SMM_NODES_RETRY;   // entries of a global pool, the most a list may hold
constexpr int SL_RETRY = -2;        // nmatch mark: redone by the general kernel's retry launch
constexpr int SL_WARPS = 15;        // target haplotypes per CTA, at most (128 registers a thread)
constexpr int SL_STAGES = 4;        // groups of rows in the ring
constexpr int SL_RUN = 16;          // sites taken with the list in registers, at most
constexpr int SL_RUN_CHUNKS = 8;    // 32-entry chunks of such a list, at most
constexpr int SL_HEAD = 2 * SL_STAGES * 8 + 16;   // barriers and the count of warps that are done
constexpr int SL_CHUNKS = 32;       // parts of a haplotype's sites, at most

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
template <bool RING> struct SlRows {
    const uint8_t *compr;
    size_t rowbytes;
    int M, group;
    const uint8_t *ring;
    size_t stage_bytes;
    uint64_t *full, *empty;
    const volatile int *ended;   // warps of the CTA that are done
    int stage;
    unsigned parity;
    const uint8_t *cur;     // the next row
    int left;               // rows left in the current group
    int site;               // rows done
    bool ok;                // no wait gave up

    __device__ __forceinline__ void open(int first) {
        stage = 0; parity = 0u; left = 0; site = first; ok = true;
        cur = ring;
    }
    // the row of site 'site'
    __device__ __forceinline__ const uint2 *next() {
        if (!RING) return reinterpret_cast<const uint2 *>(compr + (size_t)site * rowbytes);
        if (left == 0) {
            ok = ok && mbar_wait(&full[stage], parity);
            // the copy starts at the 16-byte boundary at or before the group
            cur = ring + (size_t)stage * stage_bytes + (((size_t)site * rowbytes) & 15);
            left = min(group, M - site);
        }
        const uint2 *row = reinterpret_cast<const uint2 *>(cur);
        cur += rowbytes;
        return row;
    }
    __device__ __forceinline__ void release() {
        if ((threadIdx.x & 31) == 0) mbar_arrive(&empty[stage]);
        if (++stage == SL_STAGES) { stage = 0; parity ^= 1u; }
    }
    // all lanes are done with the row last taken
    __device__ __forceinline__ void done() {
        __syncwarp();
        site++;
        if (RING && --left == 0) release();
    }
    // a warp that needs no more rows still releases those the others wait
    // for, until the last one is done ('warps' of them)
    __device__ __forceinline__ void drain(int warps) {
        if (!RING || !ok) return;
        if (left) { site += left; release(); }
        for (int polls = 0; site < M && polls < MBAR_POLLS; polls++) {
            // one lane decides for the warp: others could see the count change between them
            int go = 0;
            if ((threadIdx.x & 31) == 0) go = *ended >= warps ? 2 : (int)mbar_try(&full[stage], parity);
            go = __shfl_sync(0xffffffffu, go, 0);
            if (go == 2) return;
            if (go) { site += min(group, M - site); release(); polls = 0; }
        }
        ok = site >= M;
    }
};

struct SlState {
    int n;       // entries of the list, the root last
    int cur;     // which of the two buffers holds it
    int nres;    // matches written
    int tried;   // most elements of the buffer that were needed
    int tdst;    // start of the deepest entries (their depth: site - tdst)
    int peak, past;   // most entries at a site, before any merge: up to the chunk's last start, past it
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

// 'run' sites from m on, none of them missing, with the list in registers: 32
// entries to a chunk, R chunks, each entry's lane and register fixed for the
// run (places behind the list are kept for the roots that the sites add).
// Entries that end are emptied in place and entries that repeat an interval
// stay -- they end at the same site as the deeper ones they repeat, which
// alone report -- until the end of the run puts the list back in order.
// bits: the haplotype's alleles.  An entry costs about 27 instructions a site,
// of R independent chains, where the loop over the list in shared memory costs
// about 65 of one: 1,000 haplotypes x 5,000 sites of a 10,000-haplotype panel
// 3.0 -> 1.9 ms.
template <bool WIDE, int R, int CAP>
__device__ __forceinline__ void sl_run(SlList<WIDE, CAP> &L, SlState &s, SlRows<!WIDE> &rows, int m, int run,
                                       unsigned bits, int own, int last, int K, int nwords,
                                       int4 *__restrict__ out, int cap) {
    typedef SlIv<WIDE> IV;
    typedef typename IV::T T;
    const unsigned FULL = 0xffffffffu, lt = sl_lt();
    const int lane = threadIdx.x & 31, n = s.n, end = m + run;
    T *iv = L.iv[s.cur];
    int *stp = L.st[s.cur];
    int l[R], r[R], st[R];   // empty: [1, 0]; st -1, or of a root to come
#pragma unroll
    for (int u = 0; u < R; u++) {
        const int i = 32 * u + lane;
        l[u] = 1; r[u] = 0;
        st[u] = m + (i - n) < min(end, last) ? m + (i - n) + 1 : -1;
        if (i < n) {
            const T x = iv[i];
            l[u] = IV::l(x); r[u] = IV::r(x);
            st[u] = stp[i];
        }
    }
    if (m < last) s.peak = max(s.peak, n + run);
    if (end > last) s.past = max(s.past, n + run);
    int tdst = s.tdst;
#pragma unroll 1
    for (; m < end; m++, bits >>= 1) {
        const uint2 *row = rows.next();
        if (!rows.ok) return;
        const int c0 = (int)row[nwords - 1].y;   // the row's zeros
        const bool curr = bits & 1u;
        int nl[R], nr[R];
        bool lives = false, ends = false;   // an entry among the deepest does
#pragma unroll
        for (int u = 0; u < R; u++) {
            const uint2 a = row[l[u] >> 5], b = row[r[u] >> 5];
            const int zl = (int)a.y - __popc(~a.x & (~0u << (l[u] & 31)));
            const int zr = (int)b.y - __popc(~b.x & (~1u << (r[u] & 31))) - 1;
            nl[u] = curr ? c0 + l[u] - zl : zl;
            nr[u] = curr ? c0 - 1 + r[u] - zr : zr;
            const bool deep = st[u] == tdst, alive = nl[u] <= nr[u];
            lives |= deep && alive;
            ends |= deep && !alive;
        }
        lives = __any_sync(FULL, lives);
        ends = __any_sync(FULL, ends);
        if (ends || !lives) {
            int newcount = 0;
            if (ends && tdst > own && tdst < m) {
#pragma unroll
                for (int u = 0; u < R; u++) {
                    const bool d = st[u] == tdst && nl[u] > nr[u];
                    const unsigned bd = __ballot_sync(FULL, d);
                    if (d) {
                        const int pos = s.nres + newcount + __popc(bd & lt);
                        if (pos < cap) out[pos] = make_int4(tdst, m, l[u], r[u]);
                        else s.err |= EIMP_ERR_MATCH_OVERFLOW;
                    }
                    newcount += __popc(bd);
                }
                s.tried = max(s.tried, s.nres + newcount);
            }
            if (!lives) {   // set-maximal (TargetImp.cpp:132-136)
                if (newcount && s.nres + newcount <= cap) {
                    if (newcount > 1) sl_reverse(out, s.nres, newcount);
                    s.nres += newcount;
                }
                int minst = INT_MAX;
#pragma unroll
                for (int u = 0; u < R; u++)
                    if (nl[u] <= nr[u]) minst = min(minst, st[u]);
                for (int o = 16; o; o >>= 1) minst = min(minst, __shfl_xor_sync(FULL, minst, o));
                tdst = min(minst, m < last ? m + 1 : INT_MAX);
            }
        }
#pragma unroll
        for (int u = 0; u < R; u++) {
            const bool alive = nl[u] <= nr[u];
            l[u] = alive ? nl[u] : 1;
            r[u] = alive ? nr[u] : 0;
            if (u + 2 < R) {
                if (!alive) st[u] = -1;
            } else {   // where the roots are
                if (!alive && st[u] <= m) st[u] = -1;
                if (st[u] == m + 1) { l[u] = 0; r[u] = K - 1; }
            }
        }
        rows.done();
    }
    int kept = 0;
    T carry = IV::pack(1, 0);
#pragma unroll
    for (int u = 0; u < R; u++) {
        const bool alive = l[u] <= r[u];
        const T v = IV::pack(l[u], r[u]);
        const unsigned ba = __ballot_sync(FULL, alive), below = ba & lt;
        T p = __shfl_sync(FULL, v, below ? 31 - __clz((int)below) : 0);
        if (!below) p = carry;
        const bool keep = alive && p != v;
        const unsigned bk = __ballot_sync(FULL, keep);
        if (keep) {
            const int q = kept + __popc(bk & lt);
            iv[q] = v;
            stp[q] = st[u];
        }
        if (ba) carry = __shfl_sync(FULL, v, 31 - __clz((int)ba));
        kept += __popc(bk);
    }
    s.n = kept;
    s.tdst = tdst;
    __syncwarp();
}

// The sites from m on of one haplotype on a list of CAP entries: the matches
// that start in (own, last], to where the last of them ends.  Returns M + 1
// when it is done or failed (s.err), or -- with can_switch -- the first site
// that could outgrow the list, before touching it.
template <bool WIDE, int CAP>
__device__ __forceinline__ int sl_sites(SlList<WIDE, CAP> &L, SlState &s, SlRows<!WIDE> &rows, int m, int own, int last,
                                        bool can_switch, int K,
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
    for (; m < M && s.n; m++) {
        if (can_switch && 2 * s.n + 1 > CAP) return m;
        if ((m & 31) == 0 && m != m0) {
            missw = __ballot_sync(FULL, nextg == 3);
            currw = nexth;
            nextg = m + 32 + lane < M ? g[m + 32 + lane] : 0;
            nexth = m + 32 < M ? hw[(m >> 5) + 1] : 0u;
        }
        const bool missing = (missw >> (m & 31)) & 1u;
        if (!missing) {   // a run of sites without a missing one, of those read together
            const unsigned w = missw >> (m & 31);
            const int run = min(min(w ? __ffs((int)w) - 1 : 32 - (m & 31), SL_RUN), M - m);
            const int chunks = (s.n + run + 31) / 32;
            if (chunks <= SL_RUN_CHUNKS && s.n + run < CAP) {
                const unsigned bits = currw >> (m & 31);
#define SL_CASE(R) case R: sl_run<WIDE, R, CAP>(L, s, rows, m, run, bits, own, last, K, nwords, out, cap); break
                switch (chunks) {
                    SL_CASE(1);
                    SL_CASE(2);
                    SL_CASE(3);
                    SL_CASE(4);
                    SL_CASE(5);
                    SL_CASE(6);
                    SL_CASE(7);
                default:
                    sl_run<WIDE, SL_RUN_CHUNKS, CAP>(L, s, rows, m, run, bits, own, last, K, nwords, out, cap);
                }
#undef SL_CASE
                if (!rows.ok) { s.err |= EIMP_ERR_WAIT; return M + 1; }
                m += run - 1;
                continue;
            }
        }
        const bool curr = (currw >> (m & 31)) & 1u;
        const uint2 *row = rows.next();
        if (!rows.ok) { s.err |= EIMP_ERR_WAIT; return M + 1; }
        const int c0 = (int)row[nwords - 1].y;   // the row's zeros
        const bool hastd = s.tdst < m;           // an entry deeper than the root exists
        const bool emit = s.tdst > own;          // the deepest entries' matches belong here
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
                const unsigned ba = __ballot_sync(FULL, alive), bd = __ballot_sync(FULL, emit && deep && !alive);
                const unsigned below = ba & lt;
                T p = __shfl_sync(FULL, v, below ? 31 - __clz((int)below) : 0);
                if (!below) p = carry;
                const bool keep = alive && p != v;
                const unsigned bk = __ballot_sync(FULL, keep);
                if (emit && deep && !alive) {
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
                        dead = ext && emit && deep && !a0 && !a1;
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
        s.tried = max(s.tried, s.nres + newcount);
        const bool root = m < last;   // the next chunk has the later starts
        if (root) s.peak = max(s.peak, alln);
        else s.past = max(s.past, alln);
        if (root && lane == 0) { iv[kept] = IV::pack(0, K - 1); st[kept] = m + 1; }
        s.n = kept + (root ? 1 : 0);
        if (!__any_sync(FULL, anydeep)) {
            // the deepest entries end here: set-maximal (TargetImp.cpp:132-136)
            if (newcount && s.nres + newcount <= cap) {
                if (newcount > 1) sl_reverse(out, s.nres, newcount);
                s.nres += newcount;
            }
            for (int o = 16; o; o >>= 1) minst = min(minst, __shfl_xor_sync(FULL, minst, o));
            s.tdst = min(minst, root ? m + 1 : INT_MAX);
        }
        rows.done();
    }
    // TargetImp.cpp:144: the erase pass, the deepest entries report
    if (s.tdst < M && s.tdst > own && m >= M) {
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

// One chunk's results in the first element of its part of the match buffer,
// until the parts are joined: matches, most entries (in its sites, past them in
// the upper half), first site not read, error (with the elements it needed on
// top of its matches in the upper half).
__device__ __forceinline__ int sl_chunk_site(int M, int chunks, int c) { return (int)((long long)M * c / chunks); }

template <bool WIDE>
__global__ void __launch_bounds__((SL_WARPS + 1) * 32) smm_list_kernel(
    const uint32_t *__restrict__ compr, int M, int K, const uint64_t *__restrict__ phased, int wM,
    const uint8_t *__restrict__ gt, int nhaps, const int32_t *__restrict__ hapmap, int4 *__restrict__ matches, int cap,
    int *__restrict__ nmatch, uint32_t *__restrict__ status, int warps, int group, unsigned stage_bytes,
    SlList<WIDE, SL_POOL> *__restrict__ gpool, int gpool_slots, int *__restrict__ gpool_next, int chunks = 1) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    constexpr bool RING = !WIDE;   // rows of a wide panel are read in place
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int h0 = blockIdx.x * warps, chunk = blockIdx.y;
    const int live = min(warps, nhaps - h0);   // haplotypes of this CTA
    const int nwords = (K + 31) / 32;
    const int first = sl_chunk_site(M, chunks, chunk), last = sl_chunk_site(M, chunks, chunk + 1);
    uint64_t *full = reinterpret_cast<uint64_t *>(smem_raw), *empty = full + SL_STAGES;
    int *ended = reinterpret_cast<int *>(empty + SL_STAGES);
    uint8_t *ring = smem_raw + SL_HEAD;
    SlList<WIDE, SL_CAP> *lists =
        reinterpret_cast<SlList<WIDE, SL_CAP> *>(ring + (RING ? (size_t)SL_STAGES * stage_bytes : 0));
    SlRows<RING> rows;
    rows.compr = reinterpret_cast<const uint8_t *>(compr);
    rows.rowbytes = (size_t)nwords * 8;
    rows.M = M; rows.group = group;
    rows.ring = ring; rows.stage_bytes = stage_bytes;
    rows.full = full; rows.empty = empty; rows.ended = ended;
    if (RING) {
        if (threadIdx.x == 0) {
            for (int i = 0; i < SL_STAGES; i++) { mbar_init(&full[i], 1); mbar_init(&empty[i], live); }
            *ended = 0;
            mbar_init_fence();
        }
        __syncthreads();
        if (wid == warps) {   // the producer: one thread copies group after group until nobody reads on
            if (lane == 0) {
                const int ngroups = (M - first + group - 1) / group;
                int stage = 0, gi = 0;
                unsigned parity = 1u;   // a fresh barrier's previous phase counts as done
                bool ok = true;
                for (; gi < ngroups; gi++) {
                    int polls = 0;
                    while (!(ok = mbar_try(&empty[stage], parity)) && *(volatile int *)ended < live &&
                           ++polls < MBAR_POLLS) {}
                    if (!ok) { ok = polls < MBAR_POLLS; break; }
                    if (*(volatile int *)ended >= live) break;
                    const size_t a = (first + (size_t)gi * group) * rows.rowbytes;
                    const size_t b = min(first + (size_t)(gi + 1) * group, (size_t)M) * rows.rowbytes;
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
    // a chunk's part of the buffer: one element for its results, then its matches
    const int part = cap / chunks;
    int4 *res = matches + (size_t)hap * cap + (size_t)chunk * part;
    int4 *out = chunks > 1 ? res + 1 : res;
    if (chunks > 1) cap = part - 1;
    const unsigned FULL = 0xffffffffu;
    rows.open(first);
    // missingness > 50 %: no matches (TargetImp.cpp:79-80)
    int nmiss = 0;
#pragma unroll 4
    for (int m = lane; m < M; m += 32) nmiss += g[m] == 3;
    for (int o = 16; o; o >>= 1) nmiss += __shfl_xor_sync(FULL, nmiss, o);
    SlState s;
    s.n = 1; s.cur = 0; s.nres = 0; s.tried = 0; s.tdst = first; s.peak = 0; s.past = 0; s.err = 0u;
    const int own = chunk ? first : -1;
    if (nmiss <= M / 2) {
        SlList<WIDE, SL_CAP> &L = lists[wid];
        if (lane == 0) { L.iv[0][0] = SlIv<WIDE>::pack(0, K - 1); L.st[0][0] = first; }
        __syncwarp();
        const int m = sl_sites<WIDE, SL_CAP>(L, s, rows, first, own, last, gpool != nullptr, K, nwords, g, hw, out, cap);
        if (m <= M) {   // the list could outgrow shared memory: on in a global pool
            int slot = 0;
            if (lane == 0) slot = atomicAdd(gpool_next, 1);
            slot = __shfl_sync(FULL, slot, 0);
            if (slot < gpool_slots) {
                SlList<WIDE, SL_POOL> &G = gpool[slot];
                for (int i = lane; i < s.n; i += 32) { G.iv[0][i] = L.iv[s.cur][i]; G.st[0][i] = L.st[s.cur][i]; }
                s.cur = 0;
                __syncwarp();
                sl_sites<WIDE, SL_POOL>(G, s, rows, m, own, last, false, K, nwords, g, hw, out, cap);
            } else {
                sl_sites<WIDE, SL_CAP>(L, s, rows, m, own, last, false, K, nwords, g, hw, out, cap);
            }
        }
    }
    const int end = rows.site;
    __syncwarp();
    if (RING && lane == 0) atomicAdd(ended, 1);
    rows.drain(live);
    if (!rows.ok) s.err |= EIMP_ERR_WAIT;
    for (int o = 16; o; o >>= 1) s.err |= __shfl_xor_sync(FULL, s.err, o);
    if (lane) return;
    if (chunks > 1) { *res = make_int4(s.nres, s.peak | s.past << 16, end, (int)s.err | min(s.tried - s.nres, 0x7fff) << 16); return; }
    if (!s.err) { nmatch[hap] = s.nres; return; }
    if (s.err == EIMP_ERR_NODE_OVERFLOW) { nmatch[hap] = SL_RETRY; return; }
    nmatch[hap] = -1;
    atomicOr(status, s.err);
}

// Joins the chunks' parts of a haplotype's match buffer, one warp per
// haplotype.  A haplotype is searched again in one piece by the retry launch
// -- and accepted or refused there as a whole -- when a chunk outgrew its list
// or its part of the buffer, when the lists of the chunks that share a site
// could make one larger than the most a list may hold, or when the buffer
// would have been too small on the way.  Searching those with this kernel in one
// piece first, a pool for each, is no better throughout: 16, 64 and 200
// haplotype pairs x 3,000 sites of 20,000 haplotypes, half the genotypes of 75
// sites missing, 1.5, 13.9 and 14.7 ms without, 3.9, 11.5 and 15.8 with it (the
// general kernel alone 19, 33 and 37; without missing genotypes in bunches
// 0.45, 0.72 and 1.7).
__global__ void __launch_bounds__(32) smm_list_join_kernel(int M, const int32_t *__restrict__ hapmap,
                                                           int4 *__restrict__ matches, int cap,
                                                           int *__restrict__ nmatch, uint32_t *__restrict__ status,
                                                           int chunks) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x;
    const int hap = hapmap ? hapmap[blockIdx.x] : blockIdx.x;
    const int part = cap / chunks;
    int4 *out = matches + (size_t)hap * cap;
    int4 r = make_int4(0, 0, 0, 0);
    if (lane < chunks) r = out[(size_t)lane * part];
    const int site = sl_chunk_site(M, chunks, min(lane, chunks - 1));
    int together = 0;   // an upper bound of the entries at the sites of this lane's chunk
    int upto = 0;       // matches up to its end
    for (int c = 0; c < chunks; c++) {
        const int peak = __shfl_sync(FULL, r.y, c), end = __shfl_sync(FULL, r.z, c);
        const int k = __shfl_sync(FULL, r.x, c);
        if (c <= lane) upto += k;
        if (c == lane) together += peak & 0xffff;
        else if (c < lane && end > site) together += peak >> 16;
    }
    const bool failed = __any_sync(FULL, (r.w & EIMP_ERR_WAIT) != 0);
    const bool again = __any_sync(FULL, (r.w & 0xffff) != 0 || (lane < chunks && together > SL_POOL) ||
                                             (lane < chunks && upto + (r.w >> 16) > cap));
    if (failed || again) {
        if (lane == 0) {
            nmatch[hap] = failed ? -1 : SL_RETRY;
            if (failed) atomicOr(status, (uint32_t)EIMP_ERR_WAIT);
        }
        return;
    }
    int n = 0;
    // to the front, chunk after chunk: never past what is still to be read
    for (int c = 0; c < chunks; c++) {
        const int k = __shfl_sync(FULL, r.x, c);
        const int4 *src = out + (size_t)c * part + 1;
        for (int i0 = 0; i0 < k; i0 += 32) {
            int4 v = make_int4(0, 0, 0, 0);
            if (i0 + lane < k) v = src[i0 + lane];
            __syncwarp();
            if (i0 + lane < k) out[n + i0 + lane] = v;
            __syncwarp();
        }
        n += k;
    }
    if (lane == 0) nmatch[hap] = n;
}

// ---------------------------------------------------------------------------
// launcher
// ---------------------------------------------------------------------------
size_t smm_list_slot_bytes(int K) { return K <= 65536 ? sizeof(SlList<false, SL_POOL>) : sizeof(SlList<true, SL_POOL>); }

// A chunk is no shorter than 128 sites, about the length of a match.
int smm_list_max_chunks(int M) { return M / 128 < 1 ? 1 : M / 128 > SL_CHUNKS ? SL_CHUNKS : M / 128; }

struct SlShape { int warps, chunks, group; size_t stage, smem; };

// Chunks, haplotypes per CTA and the ring for a search.  Narrow intervals (at
// most 65,536 haplotypes, rows up to 16 KB): rows through the ring, about 8 KB
// a group, so that the haplotypes of a CTA share them.  Wide: rows in place,
// nothing shared in a CTA.
static SlShape sl_shape(int M, int K, int nhaps, int cap, int nsm, int lim, int lim_sm) {
    const bool wide = K > 65536;
    const size_t rowbytes = (size_t)((K + 31) / 32) * 8;
    const size_t list = wide ? sizeof(SlList<true, SL_CAP>) : sizeof(SlList<false, SL_CAP>);
    SlShape f;
    f.group = 0;
    f.stage = 0;
    if (!wide) {
        f.group = (int)(8192 / rowbytes);
        f.group = f.group < 1 ? 1 : f.group > 16 ? 16 : f.group;
        f.stage = (f.group * rowbytes + 30) & ~(size_t)15;   // a copy starts up to 15 bytes before its rows
    }
    const size_t head = SL_HEAD + SL_STAGES * f.stage;
    int most = (int)(((size_t)lim - head) / list);
    most = most > SL_WARPS ? SL_WARPS : most;
    if (wide && most > 4) most = 4;
    // Chunks for about 12 warps per SM.  Of 1, 4, 8, 12, 16 and 24, with three
    // batches in flight: 400 haplotypes x 2,000 sites 0.50, 0.41, 0.47, 0.40,
    // 0.45, 0.51 ms; 128 x 3,000 1.40, 1.25, 1.02, 1.03, 1.11, 1.52 ms (with
    // 1,000 haplotypes it is one chunk up to 12, and two are 4 % slower).  With
    // at least 64 or 256 sites instead of 128 there is no difference beyond
    // the spread, but longer ones leave warps out.
    long long chunks = (long long)12 * nsm / nhaps;
    if (chunks > smm_list_max_chunks(M)) chunks = smm_list_max_chunks(M);
    if (chunks > cap / 16) chunks = cap / 16;
    for (f.chunks = (int)chunks; f.chunks > 1; f.chunks--)
        for (f.warps = 1; f.warps <= most; f.warps++) {
            f.smem = head + f.warps * list;
            int per_sm = (int)(lim_sm / (f.smem + 1024));   // 1 KB of a CTA's shared memory is the system's
            const int ctas = (nhaps + f.warps - 1) / f.warps;
            if ((long long)ctas * f.chunks <= (long long)per_sm * nsm) return f;
        }
    f.chunks = 1;
    f.warps = (nhaps + nsm - 1) / nsm;
    if (f.warps > most) {
        const int waves = (nhaps + most * nsm - 1) / (most * nsm);
        f.warps = wide ? most : (nhaps + waves * nsm - 1) / (waves * nsm);
    }
    f.smem = head + f.warps * list;
    return f;
}

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
    int lim_sm = 0;
    e = cudaDeviceGetAttribute(&lim_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev);
    if (e != cudaSuccess) return e;
    const SlShape f = sl_shape(M, K, nhaps, cap, nsm, lim, lim_sm);
    if ((e = ensure_dynamic_smem((const void *)smm_list_kernel<WIDE>, f.smem)) != cudaSuccess) return e;
    smm_list_kernel<WIDE><<<dim3((nhaps + f.warps - 1) / f.warps, f.chunks), (f.warps + (f.group ? 1 : 0)) * 32, f.smem, st>>>(
        compr, M, K, phased, wM, gt, nhaps, hapmap, matches, cap, nmatch, status, f.warps, f.group, (unsigned)f.stage,
        static_cast<SlList<WIDE, SL_POOL> *>(gpool), gpool_slots, gpool_next, f.chunks);
    if (f.chunks > 1)
        smm_list_join_kernel<<<nhaps, 32, 0, st>>>(M, hapmap, matches, cap, nmatch, status, f.chunks);
    return launched(f.chunks > 1 ? 2 : 1);
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
