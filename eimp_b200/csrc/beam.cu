// Eagle2-style beam phasing over the condensed PBWT, one CTA per target.
//
// Device restatement of Target::phaseExtPBWT (Target.cpp:291-777) with Beam
// (Beam.cpp:41-837), BeamPath (BeamPath.cpp:29-291), HaplotypePath
// (HaplotypePath.cpp:36-483), BooleanHistory (BooleanHistory.cpp:31-113),
// History (History.h:29-81) and MinMaxHeap (MinMaxHeap.h:29-214).
//
// What bounds it: the chain of beam steps.  A target takes one step per split
// site and direction, each step depends on the one before, and a step holds
// few paths (on dense arrays two beam paths and four haplotype paths at the
// median), so what counts is the latency of a step, and that is the number of
// instructions of its longest thread: a warp alone takes four to five cycles
// for each.
//
// Work split inside the CTA (one target):
//  * the haplotype-path extensions (the PBWT interval mappings over the
//    history, the bulk of the work) are dealt out to all warps, a path to a
//    warp, the history steps to its lanes.  That is possible because an
//    interval list is nested -- entry i holds the haplotypes that match the
//    last i + 1 history entries -- so an extension that is empty at a step is
//    empty at all later ones: every step is mapped on its own and the lengths
//    are counts of non-empty steps.  Each step leaves its probability terms in
//    shared memory; then one lane per extension adds them in the reference's
//    order.  The reference copies intervals from the previously extended path
//    (HaplotypePath.cpp:330-390); they are recomputed here, which gives the
//    same intervals: an interval depends only on the recent history the two
//    paths share;
//  * the first warp runs the beam; the others compute the next step's
//    recombination probabilities, fetch its PBWT rows and copy the paths that
//    split while it does;
//  * with at most 32 beam paths and 32 haplotype paths a lane holds its beam
//    path's extensions in registers and sets of haplotype paths are bit masks;
//    larger beams go through shared memory, 32 at a time;
//  * the new list orders (haplotype paths after applying, beam paths after
//    applying and merging) are computed with warp scans; the positions are
//    the ones the reference's sequential loops produce;
//  * what depends on the sequential order stays on lane 0: the min-max heap
//    of the pruning, the merge of beam paths that share both histories (only
//    the duplicates, in list order), and the float sums of the calls.
// Floating point follows the reference operation by operation: float
// arithmetic with explicit double where the reference promotes (pow(), double
// literals, std::ilogb), explicit round-to-nearest intrinsics (no FMA).
//
// The beam, the lists and the target's scalars live in shared memory, and so
// do the haplotype paths (record, probability ring, three interval buffers:
// its own and its two extensions) in the first ArenaLayout::NS slots, as many
// as the launch leaves room for; the slots past them lie in the target's
// arena in global memory.  Free slots are taken lowest first, so a beam of the
// usual size stays in shared memory.  The code of a step is kept in one copy
// and small (loops over 32 paths are not unrolled, rare parts are functions
// of their own): it has to stay in the instruction cache.
//
// Measured on a B200 against one warp per target with everything but the beam
// in the arena and five copies of the step's code (kernel times): one target of
// 2,000 sites, K = 1,024 8.0 -> 2.1 ms; 100 of them 11.7 -> 3.5 ms; 192 targets
// of 32,000 sites, K = 4,096 148 -> 48 ms; 96 of 10,000 sites, K = 8,192 83 ->
// 27 ms; 1,000 of 5,000 sites, whose beams outgrow shared memory, 64 -> 55 ms.
#include <climits>

#include "async_copy.cuh"
#include "common.cuh"
#include "kernels.h"

namespace eimp {

namespace {

enum { C_HOMREF = 0, C_HETKEEP = 1, C_HETSWITCH = 2, C_HOMALT = 3, C_NONE = 4 };

struct Cons { int type, refidx; };

constexpr int PHMAX = 128;   // History<fp_type> ring (power of two >= H, H <= 128)
constexpr int PMAX = 128;    // largest beam width
constexpr int BPMAX = PMAX;  // beam paths held between two prunes (<= P)
constexpr int LMAX = 2 * PMAX + 8;   // haplotype paths in the list: each is held by a beam path's side
constexpr int HTS_BITS = 8;
constexpr int HTS = 1 << HTS_BITS;   // merge hash table entries (load <= 1/2)
static_assert(BPMAX < HTS, "the merge table must never fill");
constexpr int WITEMS = 256;  // (path, step) items of a walk whose terms a warp holds at once
constexpr int FWORDS = (4 * PMAX + 8 + 31) / 32;   // words of the free-slot mask
static_assert(FWORDS <= 32, "a lane stores a word of it");

struct HPh {   // HaplotypePath
    unsigned long long d0, d1;   // BooleanHistory data (fill mask applied)
    int last;
    float p;
    int scaleexp;
    short niv, phstart;
    unsigned char own, x0, x1;   // which of the slot's three buffers hold its intervals and its two extensions'
};

struct BPh {   // BeamPath: what it carries from step to step
    unsigned short mat, pat;     // list positions of its haplotype paths
    float prob, weight;
    int nErr;
    float pErrPath, pErrPathp1;
};
struct BXh {   // BeamPath: the extensions of the current step
    float extp[4];
    unsigned char act;           // active extensions
    signed char actidx;          // -1..3
    signed char mark;            // merging: 1 = pending, -1 = alive, -2 = erased
};

struct Hel { float key; int a; int b; };

struct Job { short src, buf, dst, n, start, pad; float p; };   // a copy of a path that splits

enum { CMD_WALK, CMD_NEXT, CMD_MEET, CMD_EXIT };   // what the other warps are to do

struct __align__(16) WS {   // a target's state in shared memory
    float scr[1056];              // the first warp's walk terms; the reference counts, the call terms or the merge table
    float prec[2][PHMAX];         // recombination probabilities of this step and the next
    BPh bp[2][BPMAX];             // the beam in list order (two buffers)
    BXh bx[BPMAX];
    // per haplotype path in list order: its slot, the extensions wanted, and
    // the extensions of this step: probabilities, scale, list lengths, active
    float ep[2][LMAX];
    int ese[LMAX];
    short happ[LMAX], happ_old[LMAX], nx[2][LMAX];
    unsigned char tox[2][LMAX], hact[LMAX];
    short2 hapmap[LMAX];          // list position of a path's two extensions
    Job job[BPMAX];
    unsigned char delmask[BPMAX]; // extensions the pruning deleted, per beam path
    unsigned fm[FWORDS];          // free slots
    Hel *heap;                    // the pruning's fallback heap: PMAX + 2 entries in the arena
    int cmd[2];
    int cursor, reverse;
    int nbp, bpsel, nhap, njob, err, qi;
    int H, P, Delta, phsize;
    unsigned long long fill0, fill1;
    int histlast;
    int ires;
    int wse, delerr;   // weightScaleExp and deleteErr of the last prune (Beam.cpp:673-678)
    int step;          // steps taken since the beam started (-1: none)
    const Cons *constr;           // per split site; null: none but the first backward step's
    short *canon;                 // per list position: first position of its run of equal histories
};

struct Ctx {
    int wid, warps;              // this warp, and the warps of the target
    float *term;                 // this warp's walk terms: two runs of WITEMS
    // haplotype paths: slots below NS in shared memory, the others in the arena
    HPh *hps, *hpg;
    float *phs, *phg;
    uint32_t *ivs, *ivg;         // intervals [l, r] packed l | r << 16 (K <= 65536)
    int NS, NR, NH, HS, HG, PHS;   // slots and records in shared memory; buffer strides (shared, arena), ring stride
    float *cdb;                  // history distances of 32 steps, [entry][step]
    // pbwt of this target: its rows, and the ring of row pairs
    const uint32_t *rows;
    uint32_t *ring;
    int nring;
    int Mp, K, kw;
    float Kinv;
    // condensed target
    const float *cmd;
    int S;
    const int32_t *calls;
    const uint8_t *tg;
    float pErr, pLimit, expectIBDcM;
    __device__ __forceinline__ HPh &hp(int slot) const { return slot < NR ? hps[slot] : hpg[slot]; }
    __device__ __forceinline__ float *ph(int slot) const {
        return slot < NS ? phs + slot * PHS : phg + (size_t)slot * PHMAX;
    }
    __device__ __forceinline__ uint32_t *iv(int slot, int which) const {
        return slot < NS ? ivs + (3 * slot + which) * HS : ivg + (size_t)(3 * slot + which) * HG;
    }
};

__device__ __forceinline__ int lane_id() { return threadIdx.x & 31; }
__device__ __forceinline__ unsigned lanemask_lt() { return (1u << (threadIdx.x & 31)) - 1u; }

// warp reductions
#ifdef __CUDACC__
__device__ __forceinline__ unsigned warp_or(unsigned v) { return __reduce_or_sync(0xffffffffu, v); }
__device__ __forceinline__ int warp_mini(int v) { return __reduce_min_sync(0xffffffffu, v); }
__device__ __forceinline__ int warp_maxi(int v) { return __reduce_max_sync(0xffffffffu, v); }
__device__ __forceinline__ int warp_sumi(int v) { return __reduce_add_sync(0xffffffffu, v); }
#else
__device__ __forceinline__ unsigned warp_or(unsigned v) {
    for (int o = 16; o; o >>= 1) v |= __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ int warp_mini(int v) {
    for (int o = 16; o; o >>= 1) v = min(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ int warp_maxi(int v) {
    for (int o = 16; o; o >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ int warp_sumi(int v) {
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
#endif
// non-negative floats order like their bit patterns
__device__ __forceinline__ float warp_maxf(float v) { return __uint_as_float((unsigned)warp_maxi((int)__float_as_uint(v))); }

// std::ilogb(float) as glibc defines it: the unbiased exponent (subnormals
// included), INT_MIN for zero and NaN, INT_MAX for infinity
__device__ __forceinline__ int ilogb_exact(float x) {
    const unsigned u = __float_as_uint(x) & 0x7fffffffu;
    if (u == 0) return INT_MIN;
    if (u >= 0x7f800000u) return u == 0x7f800000u ? INT_MAX : INT_MIN;
    const int e = (int)(u >> 23);
    if (e == 0) return (31 - __clz(u)) - 149;
    return e - 127;
}
// pow(2, n) for an integer n, as ldexp(1.0, n) gives it: the exponent field, in
// two factors where n is outside the normal range
__device__ __forceinline__ double pow2i(int n) {
    const int m = min(max(n, -2044), 2046), a = min(max(m, -1022), 1023);
    return __longlong_as_double((long long)(a + 1023) << 52) * __longlong_as_double((long long)(m - a + 1023) << 52);
}

// the same rounded to float: built from its bits in the normal range
__device__ __forceinline__ float pow2f(int n) {
    return n >= -126 && n <= 127 ? __int_as_float((n + 127) << 23) : (float)pow2i(n);
}

// ------------------------------------------------------------------ histories
__device__ __forceinline__ void bh_push(HPh &h, int b, const WS &w) {   // BooleanHistory.cpp:55-70
    unsigned long long c0 = h.d0 >> 63;
    h.d0 = (h.d0 << 1) | (unsigned long long)(b ? 1 : 0);
    h.d1 = (h.d1 << 1) | c0;
    if (h.last != w.histlast) h.last++;
    h.d0 |= w.fill0;
    h.d1 |= w.fill1;
}
__device__ __forceinline__ int bh_at(const HPh &h, int pos) {
    return (int)(((pos < 64 ? h.d0 : h.d1) >> (pos & 63)) & 1ull);
}
__device__ __forceinline__ int bh_equal(const HPh &a, const HPh &b) {
    // BooleanHistory.cpp:91-97 compares a third 8-byte slot after the data
    // words, i.e. the members 'last' and 'histlast'
    return a.d0 == b.d0 && a.d1 == b.d1 && a.last == b.last;
}

// the interval lists hold non-empty intervals of positions < K <= 65536
__device__ __forceinline__ uint32_t iv_pack(int l, int r) { return (uint32_t)l | ((uint32_t)r << 16); }
__device__ __forceinline__ int iv_l(uint32_t v) { return (int)(v & 0xffffu); }
__device__ __forceinline__ int iv_r(uint32_t v) { return (int)(v >> 16); }
// zeros of a PBWT row at the positions before i, and up to i
__device__ __forceinline__ int zeros_before(const uint2 *row, int i) {
    const uint2 p = row[i >> 5];
    return (int)p.y - __popc(~p.x & (~0u << (i & 31)));
}
__device__ __forceinline__ int zeros_upto(const uint2 *row, int i) {
    const uint2 p = row[i >> 5];
    return (int)p.y - __popc(~p.x & ~((2u << (i & 31)) - 1u));
}

// ------------------------------------------------------------------ min-max heap (MinMaxHeap.h)
__device__ __forceinline__ int hlt(const Hel &x, const Hel &y) { return x.key < y.key; }
__device__ __forceinline__ void hswap(Hel *h, int i, int j) { Hel t = h[i]; h[i] = h[j]; h[j] = t; }
__device__ __forceinline__ int hminlevel(int i) { return ((31 - __clz(i + 1)) % 2) == 0; }
__device__ __forceinline__ int hpar(int i) { return (i - 1) / 2; }

__device__ void heap_bubble_helper(Hel *h, int i, int ismax) {
    while (i != 0) {
        int p = hpar(i);
        if (p == 0) return;
        int g = hpar(p);
        if (hlt(h[i], h[g]) ^ ismax) { hswap(h, g, i); i = g; }
        else return;
    }
}
__device__ void heap_push(Hel *h, int &n, float key, int a, int b) {
    h[n].key = key; h[n].a = a; h[n].b = b;
    int i = n++;
    if (i == 0) return;
    int p = hpar(i);
    if (hminlevel(i)) {
        if (hlt(h[p], h[i])) { hswap(h, p, i); heap_bubble_helper(h, p, 1); }
        else heap_bubble_helper(h, i, 0);
    } else {
        if (hlt(h[i], h[p])) { hswap(h, p, i); heap_bubble_helper(h, p, 0); }
        else heap_bubble_helper(h, i, 1);
    }
}
__device__ void heap_trickle(Hel *h, int n, int i) {
    const int ismax = hminlevel(i) ? 0 : 1;
    while (true) {
        int ext = i, lc = 2 * i + 1;
        if (lc < n && (hlt(h[lc], h[ext]) ^ ismax)) ext = lc;
        if (lc + 1 < n && (hlt(h[lc + 1], h[ext]) ^ ismax)) ext = lc + 1;
        int lg = 2 * lc + 1;
        for (int k = 0; k < 4 && lg + k < n; ++k)
            if (hlt(h[lg + k], h[ext]) ^ ismax) ext = lg + k;
        if (i == ext) return;
        hswap(h, i, ext);
        if (ext - lc > 1) {
            if (hlt(h[hpar(ext)], h[ext]) ^ ismax) hswap(h, hpar(ext), ext);
            i = ext;
        } else return;
    }
}
__device__ Hel heap_popmin(Hel *h, int &n) {
    Hel e = h[0];
    if (n == 1) { n = 0; return e; }
    hswap(h, 0, n - 1);
    n--;
    heap_trickle(h, n, 0);
    return e;
}
__device__ __forceinline__ int heap_maxidx(const Hel *h, int n) {
    if (n == 1) return 0;
    if (n == 2) return 1;
    return hlt(h[1], h[2]) ? 2 : 1;
}

// ------------------------------------------------------------------ haplotype paths
__device__ void hp_new(const Ctx &c, WS &w, int slot, int alt) {   // HaplotypePath.cpp:36-53 (lane 0)
    HPh &h = c.hp(slot);
    h.d0 = w.fill0; h.d1 = w.fill1; h.last = -1;
    bh_push(h, alt, w);
    h.p = 1.0f; h.scaleexp = 0;
    float *ph = c.ph(slot);
#pragma unroll 1
    for (int i = 0; i < w.phsize; i++) ph[i] = 0.0f;
    h.phstart = (short)(w.phsize - 1);
    ph[h.phstart] = 1.0f;
    h.niv = 0;
    h.own = 0; h.x0 = 1; h.x1 = 2;
}

// the extensions a constraint asks of a path: bit 0 / bit 1 (HaplotypePath.cpp:139-158)
__device__ __forceinline__ int hp_required(const HPh &h, const Cons &cn) {
    if (cn.type == C_NONE) return 3;
    const int hb = bh_at(h, cn.refidx);
    if ((cn.type == C_HETKEEP && hb == 0) || (cn.type == C_HETSWITCH && hb == 1) || cn.type == C_HOMREF) return 1;
    if ((cn.type == C_HETKEEP && hb == 1) || (cn.type == C_HETSWITCH && hb == 0) || cn.type == C_HOMALT) return 2;
    return 0;
}

// updateScaling (HaplotypePath.cpp:224-258): the ring entries 0 .. niv of a
// path whose probability has left 2^-20 .. 2^20
__device__ __noinline__ void scale_ring(float *ph, int start, int niv, int pm, int e) {
    const double f = pow2i(-e);
    // a full path of a history as long as the ring: entry niv is entry 0 again
    for (int i = lane_id(); i <= min(niv, pm); i += 32) {
        float *x = &ph[(i + start) & pm];
        const float y = (float)((double)*x * f);
        *x = i + pm < niv ? (float)((double)y * f) : y;
    }
    __syncwarp();
}

// one history step of a path: interval 'from' of its list mapped against the
// cursor's two rows; the extension intervals go to e0 / e1
__device__ __forceinline__ void walk_step(const uint2 *rinc, const uint2 *rref, int cnt0, uint32_t from, float ti,
                                          uint32_t *e0, uint32_t *e1, bool &v0, bool &v1, float &f0, float &f1) {
    const int cl = zeros_before(rinc, iv_l(from)), cr = zeros_upto(rinc, iv_r(from)) - 1;
    if (cl > cr) return;
    const int zl = zeros_before(rref, cl), zr = zeros_upto(rref, cr);
    const int s0 = zr - zl, s1 = cr - cl + 1 - s0;
    v0 = s0 > 0;
    v1 = s1 > 0;
    if (v0) { *e0 = iv_pack(zl, zr - 1); f0 = __fmul_rn((float)s0, ti); }
    if (v1) { *e1 = iv_pack(cnt0 + cl - zl, cnt0 + cr - zr); f1 = __fmul_rn((float)s1, ti); }
}

// HaplotypePath::extend with updateScaling and calculateHaplotypeProbabilities
// (HaplotypePath.cpp:162-479) of this warp's share of the paths marked for
// it (list positions wid, wid + warps, ..), against the cursor's two PBWT rows.
// Step 0 is the whole row, step i maps interval i - 1.
//
// One path: the lanes take 32 steps at a time, then lane 0 adds up the terms of
// the 0-extension and lane 1 those of the 1-extension.  Several: the steps
// of up to 32 paths are laid end to end and taken 32 at a time, an item's path
// found from the bits of the paths that start within the 32; when the terms
// of WITEMS items are held (a path has at most 127), each path's lane adds
// its own.
__device__ __forceinline__ void beam_walk(const Ctx &c, WS &w) {
    const int lane = lane_id();
    const unsigned FULL = 0xffffffffu;
    const uint2 *rinc = reinterpret_cast<const uint2 *>(c.ring + (size_t)(w.step % c.nring) * 2 * c.kw);
    const uint2 *rref = rinc + c.kw / 2;
    const int nhap = w.nhap, pm = w.phsize - 1, K = c.K, H = w.H;
    const int cnt0 = (int)rref[c.kw / 2 - 1].y;   // the row's zeros
    const float *prec = w.prec[w.step & 1];
    const float prec0 = prec[0];
    float *term0 = c.term, *term1 = c.term + WITEMS;
    if (nhap <= c.wid + c.warps) {   // one path, or none
        const int q = c.wid;
        if (q >= nhap) return;
        const int t0 = w.tox[0][q], t1 = w.tox[1][q];
        if (!(t0 | t1)) return;
        const int id = w.happ[q];
        const HPh &h = c.hp(id);
        const int ps = h.phstart, niv = h.niv, lim = min(H, niv + 1);
        float *ph = c.ph(id);
        const uint32_t *iv = c.iv(id, h.own);
        uint32_t *e0 = c.iv(id, h.x0), *e1 = c.iv(id, h.x1);
        int ns = h.scaleexp;
        const int e = ilogb_exact(h.p);
        if (abs(e) >= 20) {
            ns += e;
            scale_ring(ph, ps, niv, pm, e);
        }
        int n0 = 0, n1 = 0;
#pragma unroll 1
        for (int base = 1; base < lim; base += 64) {   // two steps per lane, their lookups side by side
            bool v0[2], v1[2];
            float f0[2], f1[2];
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const int i = base + 32 * u + lane;
                v0[u] = v1[u] = false;
                f0[u] = f1[u] = 0.0f;
                if (i < lim)
                    walk_step(rinc, rref, cnt0, iv[i - 1], __fmul_rn(ph[(i + ps) & pm], prec[i]), e0 + i, e1 + i, v0[u],
                              v1[u], f0[u], f1[u]);
            }
#pragma unroll
            for (int u = 0; u < 2; u++) {
                term0[base + 32 * u + lane - 1] = f0[u];
                term1[base + 32 * u + lane - 1] = f1[u];
                n0 += __popc(__ballot_sync(FULL, v0[u]));
                n1 += __popc(__ballot_sync(FULL, v1[u]));
            }
        }
        __syncwarp();
        if (lane < 2) {   // the terms past a list's end are zeros, which leave a sum as it is
            const int cnt = lane ? K - cnt0 : cnt0, n = lane ? n1 : n0;
            const float4 *t = reinterpret_cast<const float4 *>(lane ? term1 : term0);
            float p = 0.0f;
            if (cnt > 0) {
                p = __fmul_rn((float)cnt, __fmul_rn(ph[ps & pm], prec0));
                (lane ? e1 : e0)[0] = lane ? iv_pack(cnt0, K - 1) : iv_pack(0, cnt0 - 1);
            }
#pragma unroll 1
            for (int i = 0; i < n; i += 8) {
                const float4 x = t[i >> 2], y = t[(i >> 2) + 1];
                p = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(p, x.x), x.y), x.z), x.w);
                p = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(p, y.x), y.y), y.z), y.w);
            }
            w.ep[lane][q] = (lane ? t1 : t0) ? p : 0.0f;
            w.nx[lane][q] = (short)(n + (cnt > 0));
            if (lane == 0) w.ese[q] = ns;
        }
        __syncwarp();
        return;
    }
    const unsigned le = lanemask_lt() | (1u << lane);
#pragma unroll 1
    for (int q0 = c.wid; q0 < nhap; q0 += 32 * c.warps) {
        const int q = q0 + lane * c.warps;
        int calc = 0, id = 0, ps = 0, niv = 0, bufs = 0, ns = 0, e = 0;
        if (q < nhap) {
            calc = w.tox[0][q] | w.tox[1][q] << 1;
            id = w.happ[q];
            const HPh &h = c.hp(id);
            ps = h.phstart; niv = h.niv; ns = h.scaleexp;
            bufs = (int)h.own | (int)h.x0 << 2 | (int)h.x1 << 4;
            e = ilogb_exact(h.p);
        }
        const bool sc = calc && abs(e) >= 20;
        if (sc) ns += e;
        unsigned sm = __ballot_sync(FULL, sc);
#pragma unroll 1
        while (sm) {
            const int k = __ffs((int)sm) - 1;
            sm &= sm - 1;
            scale_ring(c.ph(__shfl_sync(FULL, id, k)), __shfl_sync(FULL, ps, k), __shfl_sync(FULL, niv, k), pm,
                       __shfl_sync(FULL, e, k));
        }
        const int steps = calc ? min(H, niv + 1) - 1 : 0;
        float p0 = 0.0f, p1 = 0.0f;
        int n0 = 0, n1 = 0;
        if (calc) {   // step 0
            const float t0 = __fmul_rn(c.ph(id)[ps & pm], prec0);
            if (cnt0 > 0) {
                p0 = __fmul_rn((float)cnt0, t0);
                c.iv(id, (bufs >> 2) & 3)[0] = iv_pack(0, cnt0 - 1);
                n0 = 1;
            }
            if (cnt0 < K) {
                p1 = __fmul_rn((float)(K - cnt0), t0);
                c.iv(id, bufs >> 4)[0] = iv_pack(cnt0, K - 1);
                n1 = 1;
            }
        }
        const int items = max(steps, 1);   // an idle item where a path has no steps, or is not there
        int incl = items;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(FULL, incl, o);
            if (lane >= o) incl += y;
        }
        const unsigned pk = (unsigned)id | (unsigned)ps << 10 | (unsigned)bufs << 18;
        const int np = min(32, (nhap - q0 + c.warps - 1) / c.warps);   // paths of this round
#pragma unroll 1
        for (int first = 0; first < np;) {
            const int before = first ? __shfl_sync(FULL, incl, first - 1) : 0;
            const bool in = lane < np && lane >= first && incl - before <= WITEMS;
            const int cnt = __popc(__ballot_sync(FULL, in));
            const int tot = __shfl_sync(FULL, incl, first + cnt - 1) - before;
            const int o = incl - items - before;
            int seen = first, m0 = 0, m1 = 0;
#pragma unroll 1
            for (int base = 0; base < tot; base += 32) {
                const unsigned rel = (unsigned)(o - base);
                const unsigned starts = warp_or(in && rel < 32u ? 1u << rel : 0u);
                const int r = seen + __popc(starts & le) - 1;
                seen += __popc(starts);
                const unsigned d = __shfl_sync(FULL, pk, r);
                const int i = base + lane - __shfl_sync(FULL, o, r) + 1, lim = __shfl_sync(FULL, steps, r);
                bool v0 = false, v1 = false;
                float f0 = 0.0f, f1 = 0.0f;
                if (base + lane < tot && i <= lim) {
                    const int slot = (int)(d & 1023u);
                    uint32_t *b0 = c.iv(slot, 0);
                    const int st = slot < c.NS ? c.HS : c.HG;
                    walk_step(rinc, rref, cnt0, b0[((int)(d >> 18) & 3) * st + i - 1],
                              __fmul_rn(c.ph(slot)[(i + (int)((d >> 10) & 255u)) & pm], prec[i]),
                              b0 + ((int)(d >> 20) & 3) * st + i, b0 + ((int)(d >> 22) & 3) * st + i, v0, v1, f0, f1);
                }
                term0[base + lane] = f0;
                term1[base + lane] = f1;
                const unsigned b0 = __ballot_sync(FULL, v0), b1 = __ballot_sync(FULL, v1);
                if (in) {   // this lane's items within the 32
                    const int lo = max(o - base, 0), hi = min(o + items - base, 32);
                    if (lo < hi) {
                        const unsigned seg = (FULL >> (32 - hi)) & (FULL << lo);
                        m0 += __popc(b0 & seg);
                        m1 += __popc(b1 & seg);
                    }
                }
            }
            __syncwarp();
            if (in && calc) {   // the terms past a list's end are zeros, which leave a sum as it is
                const int n = max(m0, m1);
                const float *a = term0 + o, *b = term1 + o;
#pragma unroll 4
                for (int k = 0; k < n; k++) {
                    p0 = __fadd_rn(p0, a[k]);
                    p1 = __fadd_rn(p1, b[k]);
                }
                n0 += m0;
                n1 += m1;
            }
            __syncwarp();
            first += cnt;
        }
        if (calc) {
            w.ep[0][q] = calc & 1 ? p0 : 0.0f;
            w.ep[1][q] = calc & 2 ? p1 : 0.0f;
            w.nx[0][q] = (short)n0;
            w.nx[1][q] = (short)n1;
            w.ese[q] = ns;
        }
        __syncwarp();
    }
}

// (short code on purpose: a job in flight at a time and no unrolled copies; with
// two jobs side by side, four times the code, 1,000 targets of 5,000 sites took
// 64 instead of 59 ms a pass, three CTAs per SM fetching their instructions)
// the paths that split: this warp's share of the copies of rings (with the
// copy's own entry pushed) and extension-1 intervals
__device__ __forceinline__ void beam_copy(const Ctx &c, const WS &w, int first, int stride) {
    const int lane = lane_id(), phs = w.phsize;
#pragma unroll 1
    for (int k = first; k < w.njob; k += stride) {
        const Job &j = w.job[k];
        const float *a = c.ph(j.src);
        const uint32_t *s = c.iv(j.src, j.buf);
        float *b = c.ph(j.dst);
        uint32_t *d = c.iv(j.dst, 0);
        const int start = j.start, n = j.n;
        const float p = j.p;
#pragma unroll 1
        for (int i = lane; i < max(phs, n); i += 64) {   // two words of each per lane in flight
            float x[2];
            uint32_t v[2];
#pragma unroll
            for (int u = 0; u < 2; u++) {
                if (i + 32 * u < phs) x[u] = a[i + 32 * u];
                if (i + 32 * u < n) v[u] = s[i + 32 * u];
            }
#pragma unroll
            for (int u = 0; u < 2; u++) {
                if (i + 32 * u < phs) b[i + 32 * u] = i + 32 * u == start ? p : x[u];
                if (i + 32 * u < n) d[i + 32 * u] = v[u];
            }
        }
    }
}

// ------------------------------------------------------------------ beam paths
// the extensions a genotype is inconsistent with, as bits (BeamPath.cpp:246-274)
__device__ __forceinline__ unsigned incon_mask(int g) { return g == 1 ? 9u : g == 0 ? 14u : g == 2 ? 7u : 15u; }
__device__ __forceinline__ void bp_update_errors(BPh &b, int incon, int delerr, float pErr) {   // BeamPath.cpp:209-228
    const int add = incon - (delerr ? 1 : 0);   // -1, 0 or 1
    b.nErr += add;
    if (add < 0) { b.pErrPathp1 = b.pErrPath; b.pErrPath = __fdiv_rn(b.pErrPath, pErr); }
    else if (add > 0) { b.pErrPath = b.pErrPathp1; b.pErrPathp1 = __fmul_rn(b.pErrPathp1, pErr); }
}
__device__ __forceinline__ int top_ext(unsigned act) { return 31 - __clz((int)act); }   // -1: none

// BeamPath::extend (BeamPath.cpp:121-197): the probabilities of the extensions
// the constraint allows (mask returned), from the list positions' results
__device__ __forceinline__ unsigned bp_extend(const Ctx &c, const WS &w, const BPh &b, int g, const Cons &cn,
                                              int bpscaleexp, float (&x)[4]) {
    const int mat = b.mat, pat = b.pat;
    const float pm0 = w.ep[0][mat], pm1 = w.ep[1][mat], pp0 = w.ep[0][pat], pp1 = w.ep[1][pat];
    const float scale = pow2f(w.ese[mat] + w.ese[pat] + bpscaleexp);
    unsigned act = 15u;
    if (cn.type != C_NONE) {
        const unsigned c0 = w.tox[0][mat], c1 = w.tox[1][mat], d0 = w.tox[0][pat], d1 = w.tox[1][pat];
        act = (c0 & d0) | (c0 & d1) << 1 | (c1 & d0) << 2 | (c1 & d1) << 3;
        const int t = cn.type;
        if (t == C_HOMREF) act &= 1u;
        else if (t == C_HOMALT) act &= 8u;
        else act &= (bh_at(c.hp(w.happ[mat]), cn.refidx) == 0) == (t == C_HETKEEP) ? 2u : 4u;
    }
    const float e0 = b.pErrPath, e1 = b.pErrPathp1;
    const unsigned im = incon_mask(g);
    x[0] = __fmul_rn(__fmul_rn(__fmul_rn(pm0, pp0), scale), im & 1u ? e1 : e0);
    x[1] = __fmul_rn(__fmul_rn(__fmul_rn(pm0, pp1), scale), im & 2u ? e1 : e0);
    x[2] = __fmul_rn(__fmul_rn(__fmul_rn(pm1, pp0), scale), im & 4u ? e1 : e0);
    x[3] = __fmul_rn(__fmul_rn(__fmul_rn(pm1, pp1), scale), im & 8u ? e1 : e0);
    return act;
}

// BeamPath::markExtensionDeleted (BeamPath.cpp:101-112) on the beam path; the
// haplotype-path side is applied after the heap pass from delmask
__device__ __forceinline__ void bp_mark_deleted_deferred(WS &w, int it, int ext) {
    BXh &x = w.bx[it];
    x.act &= (unsigned char)~(1u << ext);
    x.actidx = (signed char)top_ext(x.act);
    w.delmask[it] |= (unsigned char)(1u << ext);
}

// ------------------------------------------------------------------ beam
// Beam::calculateRecProbs (Beam.cpp:541-573).  The distance to history entry
// i is the float sum of the i preceding split-site distances, from the cursor
// back; the sums of different steps are independent, so every 32 steps each
// lane adds up one step's, in the reference's order.  The probabilities are
// per entry (lanes), for the entries the beam's paths reach.  A double sum
// 1.0 + x or quotient 1.0 / x of floats, rounded to float, is the float
// operation's result (the double has more than twice the float's bits).
__device__ __noinline__ void rec_distances(float *cdb, const float *cmd, int cur, bool rev, int H, int S) {
    const int lane = lane_id(), lc = rev ? cur - lane : cur + lane;   // the lane's cursor
    const int L = (lc >= 0 && lc < S) ? (rev ? min(H, S - lc) : min(H, lc + 1)) : 0;
    float cd = 0.0f;
    __syncwarp();
#pragma unroll 4
    for (int i = 0; i < L; i++) {
        cdb[i * 32 + lane] = cd;
        cd = __fadd_rn(cd, cmd[rev ? lc + 1 + i : lc - i]);
    }
    __syncwarp();
}
__device__ __forceinline__ void beam_calc_rec(const Ctx &c, WS &w, int step) {
    const int lane = lane_id();
    const bool rev = w.reverse != 0;
    const int cur = rev ? c.S - 1 - step : step, k = step & 31;
    float *prec = w.prec[step & 1];
    if (k == 0) rec_distances(c.cdb, c.cmd, cur, rev, w.H, c.S);
    const int L = rev ? min(w.H, c.S - cur) : min(w.H, cur + 1);
    const float cursordiff = rev ? c.cmd[cur] : c.cmd[cur + 1];
#pragma unroll 1
    for (int i = lane; i < L; i += 32) {
        const float cd = c.cdb[i * 32 + k];
        const float tmp1 = __fadd_rn(1.0f, __fdiv_rn(cd, c.expectIBDcM));
        float pr = __fdiv_rn(1.0f, __fmul_rn(tmp1, tmp1));
        const float tmp2 = __fadd_rn(1.0f, __fdiv_rn(__fadd_rn(cd, cursordiff), c.expectIBDcM));
        pr = (float)((double)pr - 1.0 / (double)__fmul_rn(tmp2, tmp2));
        pr = fmaxf(fminf(pr, 1.0f), 0.000001f);
        prec[i] = __fmul_rn(pr, c.Kinv);
    }
}

// Copies step q's two PBWT rows (the incon row of the previous split site and
// the ref row of this one, neighbours in storage in both directions) into its
// place in the ring; every call closes a copy group, past the last step an
// empty one.
__device__ __forceinline__ void beam_copy_rows(const Ctx &c, const WS &w, int q) {
    if (q < c.S) {
        const uint32_t *src = c.rows + (size_t)((w.reverse ? c.Mp : 0) + 2 * q) * c.kw;
        uint32_t *dst = c.ring + (size_t)(q % c.nring) * 2 * c.kw;
        if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) {
#pragma unroll 1
            for (int i = lane_id(); i < c.kw / 2; i += 32) copy_async16(dst + 4 * i, src + 4 * i);
        } else {   // an odd number of words to a row
#pragma unroll 1
            for (int i = lane_id(); i < c.kw; i += 32) copy_async8(dst + 2 * i, src + 2 * i);
        }
    }
    copy_async_commit();
}

// Makes step 'step' ready (one warp): its recombination probabilities, its
// rows landed, and the copy of a later step's started.  The step before may
// still be read (it is walked again when its constraint fails): a ring of three
// prefetches two steps ahead, a ring of two the step itself.
__device__ __forceinline__ void beam_next(const Ctx &c, WS &w, int step) {
    if (step >= c.S) return;
    if (step == 0) {
        copy_async_wait<0>();   // of a beam that ended before
        __syncwarp();
#pragma unroll 1
        for (int q = 0; q < c.nring - 2; q++) beam_copy_rows(c, w, q);
    }
    beam_copy_rows(c, w, step + c.nring - 2);
    beam_calc_rec(c, w, step);
    if (c.nring == 3) copy_async_wait<1>();
    else copy_async_wait<0>();
    __syncwarp();
}

// apply the haplotype-path extensions (Beam.cpp:684-726).  The new list holds
// the paths extended with 0 in old order, then the paths extended with 1 in
// old order; a path with both extensions stays among the first and its copy
// (HaplotypePath.cpp:55-75), which takes the 1-extension, among the second.
// Positions come from warp scans; released slots are free before the copies
// take theirs, the lowest first (slot numbers are storage only and do not
// change results).
__device__ __forceinline__ void beam_apply_hap(const Ctx &c, WS &w) {
    const int lane = lane_id();
    const unsigned FULL = 0xffffffffu, lt = lanemask_lt();
    const int nold = w.nhap, pm = w.phsize - 1;
    int next0 = 0, ncp = 0;
#pragma unroll 1
    for (int base = 0; base < nold; base += 32) {
        const int i = base + lane;
        int a = 0;
        if (i < nold) {
            const int id = w.happ[i];
            w.happ_old[i] = (short)id;
            a = w.hact[i];
            if (!a) atomicOr(&w.fm[id >> 5], 1u << (id & 31));
        }
        next0 += __popc(__ballot_sync(FULL, a & 1));
        ncp += __popc(__ballot_sync(FULL, a == 3));
    }
    __syncwarp();
    if (ncp) {   // a slot for each copy
        int wi = 0, k = 0;
        unsigned f = w.fm[0];
#pragma unroll 1
        while (k < ncp) {
            if (!f) {
                if (++wi == FWORDS) break;
                f = w.fm[wi];
                continue;
            }
            if (lane == 0) w.job[k].dst = (short)(32 * wi + __ffs((int)f) - 1);
            f &= f - 1;
            k++;
        }
        __syncwarp();   // the mask changes when all lanes have read it
        if (lane < wi) w.fm[lane] = 0u;
        if (lane == wi && wi < FWORDS) w.fm[wi] = f;
        if (k < ncp) {
            if (lane == 0) w.err |= EIMP_ERR_BEAM_CAPACITY;
            __syncwarp();
            return;
        }
        __syncwarp();
    }
    int zero = 0, one = next0, cp = 0;
#pragma unroll 1
    for (int base = 0; base < nold; base += 32) {
        const int i = base + lane;
        const int a = i < nold ? (int)w.hact[i] : 0;
        const unsigned b0 = __ballot_sync(FULL, a & 1), b1 = __ballot_sync(FULL, a & 2);
        const unsigned bc = b0 & b1;
        const int z = zero + __popc(b0 & lt), o = one + __popc(b1 & lt);
        if (a) {
            w.hapmap[i] = make_short2((short)z, (short)o);
            const int id = w.happ_old[i], se = w.ese[i];
            HPh &h = c.hp(id);
            const int start = (h.phstart - 1) & pm;
            if (a == 3) {   // HaplotypePath.cpp:55-75
                Job &j = w.job[cp + __popc(bc & lt)];
                const int n1 = w.nx[1][i];
                const float p = w.ep[1][i];
                const int slot = j.dst;
                j.src = (short)id; j.buf = h.x1; j.n = (short)n1; j.start = (short)start; j.p = p;
                HPh n = h;
                bh_push(n, 1, w);
                n.p = p; n.scaleexp = se;
                n.niv = (short)n1; n.phstart = (short)start;
                n.own = 0; n.x0 = 1; n.x1 = 2;
                c.hp(slot) = n;
                w.happ[o] = (short)slot;
            }
            // HaplotypePath::applyExtension (HaplotypePath.cpp:77-103)
            const int e = a == 2;
            bh_push(h, e, w);
            const float p = w.ep[e][i];
            h.p = p; h.scaleexp = se;
            h.phstart = (short)start;
            c.ph(id)[start] = p;
            const unsigned char t = h.own;
            if (e) { h.own = h.x1; h.x1 = t; } else { h.own = h.x0; h.x0 = t; }
            h.niv = w.nx[e][i];
            w.happ[e ? o : z] = (short)id;
        }
        zero += __popc(b0); one += __popc(b1); cp += __popc(bc);
    }
    if (lane == 0) { w.nhap = one; w.njob = ncp; }
    __syncwarp();
}

// each list position's first position of its run of equal histories (runs of
// equal histories are adjacent in the list)
__device__ __forceinline__ void beam_canon(const Ctx &c, WS &w) {
    const int lane = lane_id();
    const unsigned FULL = 0xffffffffu;
    const int nhap = w.nhap;
    int carry = 0;
#pragma unroll 1
    for (int base = 0; base < nhap; base += 32) {
        const int i = base + lane;
        bool head = true;
        if (i < nhap && i > 0) head = !bh_equal(c.hp(w.happ[i]), c.hp(w.happ[i - 1]));
        const unsigned hb = __ballot_sync(FULL, i < nhap && head);
        const unsigned upto = hb & (lane == 31 ? FULL : ((2u << lane) - 1u));
        const int cn = upto ? base + 31 - __clz((int)upto) : carry;
        if (i < nhap) w.canon[i] = (short)cn;
        carry = __shfl_sync(FULL, cn, 31);
    }
    __syncwarp();
}

// A command to the other warps: they read its slot after the barrier, and the
// next command goes to the other slot.
__device__ __forceinline__ void beam_command(const Ctx &c, WS &w, int &ncmd, int cmd) {
    __syncwarp();
    if (c.warps > 1) {
        if (lane_id() == 0) w.cmd[ncmd & 1] = cmd;
        ncmd++;
        block_barrier(32 * c.warps);
    }
}

// What a command asks of this warp.  All warps walk, and meet again; then the
// second warp makes the next step ready, and the third waits for the first to
// have pruned (w.ires survivors, w.hact), applies the haplotype-path
// extensions while the first applies the beam paths', and meets it; the warps
// from the third on copy the paths that split.
__device__ __forceinline__ void beam_help(const Ctx &c, WS &w) {
    int ready = 0;   // the step made ready last
    for (int ncmd = 0;; ncmd++) {
        block_barrier(32 * c.warps);
        const int cmd = w.cmd[ncmd & 1];
        if (cmd == CMD_EXIT) return;
        if (cmd == CMD_NEXT) {
            ready = 0;
            if (c.wid == 1) beam_next(c, w, 0);
        } else if (cmd == CMD_WALK) {
            const int next = w.step + 1;
            beam_walk(c, w);
            block_barrier(32 * c.warps);
            if (next != ready) {
                ready = next;
                if (c.wid == 1) beam_next(c, w, next);
            }
            if (c.wid == 2) {   // the third warp applies the extensions that survive
                pair_barrier(1, 64);
                if (w.ires > 0) {
                    beam_apply_hap(c, w);
                    if (!w.err) beam_canon(c, w);
                    pair_barrier(2, 64);
                }
            }
            if (c.wid >= 2) {   // it and those after it copy the paths that split
                if (c.warps > 3) pair_barrier(3, 32 * (c.warps - 2));
                if (w.ires > 0 && !w.err) beam_copy(c, w, c.wid - 2, c.warps - 2);
            }
        }
        __syncwarp();
    }
}

__device__ __noinline__ void beam_init(const Ctx c, WS &w, const Cons *constr, int reverse, int H, int P, int Delta) {
    const int lane = lane_id();
    __syncwarp();
#pragma unroll 1
    for (int i = lane; i < FWORDS; i += 32) {
        const int n = c.NH - 32 * i;   // slots 0 and 1 are taken below
        w.fm[i] = (n >= 32 ? 0xffffffffu : n > 0 ? (1u << n) - 1u : 0u) & (i == 0 ? ~3u : ~0u);
    }
#pragma unroll 1
    for (int i = lane; i < PHMAX; i += 32) { w.prec[0][i] = 0.0f; w.prec[1][i] = 0.0f; }
    __syncwarp();
    if (lane == 0) {   // Beam.cpp:41-92
        w.H = H; w.P = P; w.Delta = Delta;
        int l2 = 31 - __clz(H);
        if ((1 << l2) != H) l2++;
        w.phsize = 1 << l2;
        w.histlast = H - 1;
        int lw = (H - 1) / 64;
        unsigned long long mlw = (H % 64 == 0) ? 0ull : ~((1ull << (H % 64)) - 1ull);
        w.fill0 = 0 < lw ? 0ull : (0 == lw ? mlw : ~0ull);
        w.fill1 = 1 < lw ? 0ull : (1 == lw ? mlw : ~0ull);
        w.reverse = reverse;
        w.constr = constr;
        w.cursor = reverse ? c.S : -1;
        w.step = -1;
        w.err = 0;
        hp_new(c, w, 0, 0);
        hp_new(c, w, 1, 1);
        w.happ[0] = 0; w.happ[1] = 1;
        w.nhap = 2;
        w.bpsel = 0;
        BPh &b = w.bp[0][0];
        b.mat = 0; b.pat = 1; b.weight = 1.0f;
        b.nErr = 0; b.pErrPath = 1.0f; b.pErrPathp1 = __fmul_rn(1.0f, c.pErr);
        b.prob = (float)(pow2i(0) * (double)c.hp(0).p * (double)c.hp(1).p * 1.0);
        w.nbp = 1;
    }
    __syncwarp();
}

// Beam::prunePaths (Beam.cpp:577-787), the filter and the min-max heap.  The
// candidates are, per beam path in list order, the extension indices from
// the active index down to 0 (unconstrained) or the active index alone.
//
// The reference streams the candidates at or above the limit through a
// min-max heap of capacity P that replaces its minimum only by a strictly
// larger key.  When at most P candidates reach the limit nothing is evicted;
// when more do but the P-th largest key is strictly larger than the
// (P+1)-th, the heap ends holding exactly the P largest (every candidate
// outside it is at most the final minimum, every one inside at least).  In
// both cases the lanes decide everything: the P-th largest key comes from a
// bitwise search over the keys (non-negative floats order like their bit
// patterns), and the heap's minimum and maximum are a survivor with the
// smallest and one with the largest key, provided all survivors tied at the
// smallest key give the same weightScaleExp and all tied at the largest the
// same deleteErr (else which tied element the heap holds at its root would
// matter).  Otherwise lane 0 runs the heap in the reference's order.  The
// reference counts of the haplotype paths are decremented afterwards by the
// lanes (nothing in the selection reads them).  Returns 0 when no extension
// survives.
__device__ __forceinline__ unsigned key_bits(float p) { return p == 0.0f ? 0u : __float_as_uint(p); }

// A key that exactly P of the selected candidates reach, by bisection over the
// bits below those they share; false when there is none (ties straddle the
// P-th place).  A lane's candidates are held in registers.
__device__ __noinline__ bool prune_threshold(const WS &w, unsigned sel, int nr, int P, unsigned kmin, unsigned kmax,
                                             unsigned *out) {
    const int lane = lane_id();
    unsigned k[16];
#pragma unroll
    for (int q = 0; q < 16; q++) k[q] = (sel >> q) & 1u ? key_bits(w.bx[lane + 32 * (q >> 2)].extp[q & 3]) : 0u;
    if (kmin == kmax) return false;
    const int top = 31 - __clz((int)(kmin ^ kmax));
    unsigned thr = kmin & ~((2u << top) - 1u);
#pragma unroll 1
    for (int bit = top; bit >= 0; bit--) {
        const unsigned cand = thr | (1u << bit);
        int cnt = 0;
#pragma unroll
        for (int q = 0; q < 16; q++) cnt += ((sel >> q) & 1u) && k[q] >= cand;
        cnt = warp_sumi(cnt);
        if (cnt == P) { *out = cand; return true; }
        if (cnt > P) thr = cand;
    }
    return false;
}

// the heap in the reference's order (lane 0)
__device__ __noinline__ void prune_heap(WS &w, const BPh *bp, float limit, bool allext) {
    Hel *hq = w.heap;
    const int nbp = w.nbp, P = w.P;
    int n = 0;
#pragma unroll 1
    for (int it = 0; it < nbp; it++) {
        const BXh &x = w.bx[it];
        int ex = x.actidx;
        while (ex >= 0) {
            const float p = x.extp[ex];
            if (p >= limit) {
                if (n < P || (n == P && p > hq[0].key)) {
                    if (n == P) {
                        Hel e = heap_popmin(hq, n);
                        bp_mark_deleted_deferred(w, e.a, e.b);
                    }
                    heap_push(hq, n, p, it, ex);
                } else bp_mark_deleted_deferred(w, it, ex);
            } else bp_mark_deleted_deferred(w, it, ex);
            ex = allext ? ex - 1 : -1;
        }
    }
    w.ires = n;
    if (n) {
        w.wse = -ilogb_exact(bp[hq[0].a].weight);                    // weightScaleExp
        w.delerr = bp[hq[heap_maxidx(hq, n)].a].nErr > 0;            // deleteErr
    }
}

__device__ __noinline__ int beam_prune_select(WS &w, float pLimit, float maxP, bool allext) {
    const int lane = lane_id();
    BPh *bp = w.bp[w.bpsel];
    const int nbp = w.nbp, P = w.P;
    const int nr = (nbp + 31) / 32;   // beam paths per lane
    const float limit = __fmul_rn(pLimit, maxP);
#pragma unroll 1
    for (int it = lane; it < nbp; it += 32) w.delmask[it] = 0;
    // the candidates at or above the limit: bit 4r+ex of sel for extension ex
    // of beam path lane+32r (their keys are read back from shared memory)
    unsigned sel = 0;
    unsigned kmin = 0x7f800000u, kmax = 0u;
#pragma unroll 1
    for (int r = 0; r < nr; r++) {
        const int it = lane + 32 * r;
        const BXh &x = w.bx[it < nbp ? it : 0];
        const int ai = it < nbp ? (int)x.actidx : -1;
#pragma unroll
        for (int ex = 0; ex < 4; ex++) {
            if (ex <= ai && (allext || ex == ai)) {
                const float p = x.extp[ex];
                if (p >= limit) {
                    sel |= 1u << (4 * r + ex);
                    const unsigned k = key_bits(p);
                    kmin = k < kmin ? k : kmin;
                    kmax = k > kmax ? k : kmax;
                }
            }
        }
    }
    const int nA = warp_sumi(__popc(sel));
    kmin = (unsigned)warp_mini((int)kmin);
    kmax = (unsigned)warp_maxi((int)kmax);
    // survivors: the selected candidates with key >= thr
    unsigned thr = 0u;
    bool fast = true;
    if (nA > P) fast = prune_threshold(w, sel, nr, P, kmin, kmax, &thr);   // else ties straddle the P-th place
    unsigned surv = sel;
    if (thr)
#pragma unroll 1
        for (int q = 0; q < nr * 4; q++)
            if (((sel >> q) & 1u) && key_bits(w.bx[lane + 32 * (q >> 2)].extp[q & 3]) < thr) surv &= ~(1u << q);
    int wse = 0, delerr = 0;
    const int nsurv = nA > P ? P : nA;
    if (fast && nsurv > 0) {
        unsigned kminb = kmin;
        if (nA > P) {   // the smallest survivor
            kminb = 0x7f800000u;
#pragma unroll 1
            for (int q = 0; q < nr * 4; q++)
                if ((surv >> q) & 1u) kminb = min((int)kminb, (int)key_bits(w.bx[lane + 32 * (q >> 2)].extp[q & 3]));
            kminb = (unsigned)warp_mini((int)kminb);
        }
        int lo0 = INT_MAX, hi0 = INT_MIN, lo1 = 1, hi1 = 0;
#pragma unroll 1
        for (int q = 0; q < nr * 4; q++) {
            if (!((surv >> q) & 1u)) continue;
            const int it = lane + 32 * (q >> 2);
            const unsigned kq = key_bits(w.bx[it].extp[q & 3]);
            if (kq == kminb) { const int e = -ilogb_exact(bp[it].weight); lo0 = min(lo0, e); hi0 = max(hi0, e); }
            if (kq == kmax) { const int f = bp[it].nErr > 0; lo1 = min(lo1, f); hi1 = max(hi1, f); }
        }
        lo0 = warp_mini(lo0); hi0 = warp_maxi(hi0);
        lo1 = warp_mini(lo1); hi1 = warp_maxi(hi1);
        fast = lo0 == hi0 && lo1 == hi1;
        wse = lo0;
        delerr = lo1;
    }
    __syncwarp();
    if (fast) {
#pragma unroll 1
        for (int r = 0; r < nr; r++) {
            const int it = lane + 32 * r;
            if (it >= nbp) continue;
            BXh &x = w.bx[it];
            unsigned dm = 0, act = x.act;
#pragma unroll 1
            for (int ex = x.actidx; ex >= 0; ex = allext ? ex - 1 : -1)
                if (!((surv >> (4 * r + ex)) & 1u)) { act &= ~(1u << ex); dm |= 1u << ex; }
            if (dm) {
                x.act = (unsigned char)act;
                x.actidx = (signed char)top_ext(act);
                w.delmask[it] = (unsigned char)dm;
            }
        }
        if (lane == 0) { w.ires = nsurv; w.wse = wse; w.delerr = delerr; }
    } else if (lane == 0) prune_heap(w, bp, limit, allext);
    __syncwarp();
    const int n = w.ires;
    // the deletions (HaplotypePath::markExtensionDeleted, HaplotypePath.cpp:
    // 105-109), aggregated per haplotype-path extension: a count reaches
    // zero (the extension becomes inactive) in exactly the decrement that
    // takes it from >= 1 to <= 0, however the decrements are grouped
    int *rc0 = reinterpret_cast<int *>(w.scr), *rc1 = rc0 + LMAX;
#pragma unroll 1
    for (int it = lane; it < nbp; it += 32) {
        const unsigned dm = w.delmask[it];
        if (!dm) continue;
        const int m = bp[it].mat, q = bp[it].pat;
        // mat extension 0: ext 0, 1; 1: ext 2, 3; pat extension 0: ext 0, 2; 1: ext 1, 3
        if (dm & 3u) atomicSub(&rc0[m], __popc(dm & 3u));
        if (dm & 12u) atomicSub(&rc1[m], __popc(dm & 12u));
        if (dm & 5u) atomicSub(&rc0[q], __popc(dm & 5u));
        if (dm & 10u) atomicSub(&rc1[q], __popc(dm & 10u));
    }
    __syncwarp();
    // an extension no beam path used (constraints only) stays active
#pragma unroll 1
    for (int i = lane; i < w.nhap; i += 32) {
        const int u = w.hact[i];   // bits 0, 1: wanted; bits 2, 3: used
        w.hact[i] = (unsigned char)((((u & 1) && (rc0[i] > 0 || !(u & 4))) ? 1 : 0) |
                                    (((u & 2) && (rc1[i] > 0 || !(u & 8))) ? 2 : 0));
    }
    __syncwarp();
    return n > 0;
}

// The extensions of a beam of any size into shared memory: probabilities and
// masks per beam path, the reference counts and use of the haplotype-path
// extensions; returns the largest probability.
__device__ __noinline__ float extend_general(const Ctx c, WS &w, const Cons cn, int g, int bpscaleexp) {
    const int lane = lane_id(), nbp = w.nbp;
    const BPh *bp = w.bp[w.bpsel];
    int *rc0 = reinterpret_cast<int *>(w.scr), *rc1 = rc0 + LMAX;
#pragma unroll 1
    for (int i = lane; i < w.nhap; i += 32) { rc0[i] = 0; rc1[i] = 0; }
    __syncwarp();
    float maxP = 0.0f;
#pragma unroll 1
    for (int it = lane; it < nbp; it += 32) {
        float x[4];
        const unsigned act = bp_extend(c, w, bp[it], g, cn, bpscaleexp, x);
        BXh &o = w.bx[it];
#pragma unroll
        for (int ex = 0; ex < 4; ex++) {
            const bool a = (act >> ex) & 1u;
            o.extp[ex] = a ? x[ex] : 0.0f;
            if (a && maxP < x[ex]) maxP = x[ex];
        }
        o.act = (unsigned char)act;
        o.actidx = (signed char)top_ext(act);
        const int m = bp[it].mat, q = bp[it].pat;
        if (act & 3u) atomicAdd(&rc0[m], __popc(act & 3u));
        if (act & 12u) atomicAdd(&rc1[m], __popc(act & 12u));
        if (act & 5u) atomicAdd(&rc0[q], __popc(act & 5u));
        if (act & 10u) atomicAdd(&rc1[q], __popc(act & 10u));
    }
    __syncwarp();
#pragma unroll 1
    for (int i = lane; i < w.nhap; i += 32)
        w.hact[i] = (unsigned char)(w.tox[0][i] | w.tox[1][i] << 1 | (rc0[i] > 0) << 2 | (rc1[i] > 0) << 3);
    __syncwarp();
    return warp_maxf(maxP);
}

// The same pruning for at most 32 beam paths, a path per lane, its candidates
// x / act in registers.  Returns 1 with act the survivors, 0 when there are
// none, -1 when the heap would have to decide (nothing is changed then).
__device__ __forceinline__ int prune_small(const WS &w, float limit, float weight, int nErr, const float (&x)[4],
                                           unsigned &act, int &wse, int &delerr) {
    unsigned sel = 0u, kmin = 0x7f800000u, kmax = 0u;
#pragma unroll
    for (int ex = 0; ex < 4; ex++)
        if (((act >> ex) & 1u) && x[ex] >= limit) {
            sel |= 1u << ex;
            const unsigned k = key_bits(x[ex]);
            kmin = k < kmin ? k : kmin;
            kmax = k > kmax ? k : kmax;
        }
    const int nA = warp_sumi(__popc(sel));
    if (nA == 0) return 0;
    const unsigned lo = (unsigned)warp_mini((int)kmin), hi = (unsigned)warp_maxi((int)kmax);
    const bool ismin = sel && kmin == lo, ismax = sel && kmax == hi;
    const int e = -ilogb_exact(weight);
    const int e0 = warp_mini(ismin ? e : INT_MAX), e1 = warp_maxi(ismin ? e : INT_MIN);
    const unsigned bm = __ballot_sync(0xffffffffu, ismax), be = __ballot_sync(0xffffffffu, ismax && nErr > 0);
    if (nA > w.P || e0 != e1 || (be && be != bm)) return -1;
    wse = e0;
    delerr = be != 0;
    act = sel;
    return 1;
}

__device__ __forceinline__ void bp_make(BPh &o, const BPh &b, float p, int ex, int mat, int pat, unsigned im, int wse,
                                        float wsf, int delerr, float pErr) {   // BeamPath.cpp:44-96
    o.mat = (unsigned short)mat; o.pat = (unsigned short)pat;
    o.prob = p; o.weight = b.weight;
    o.nErr = b.nErr; o.pErrPath = b.pErrPath; o.pErrPathp1 = b.pErrPathp1;
    // weightScaleExp: exact in double, then rounded once; one float product gives
    // the same where the factor is a normal float
    if (wse != 0) o.weight = abs(wse) <= 126 ? __fmul_rn(o.weight, wsf) : (float)((double)o.weight * pow2i(wse));
    bp_update_errors(o, (int)((im >> ex) & 1u), delerr, pErr);
}

// apply the beam-path extensions (Beam.cpp:728-779): each path with a
// surviving extension keeps its position with its lowest extension; its other
// extensions are appended in the reference's order (paths in list order,
// extensions in descending index).  Positions come from warp scans.
__device__ __forceinline__ void beam_apply_bp(const Ctx &c, WS &w, int g, int wse, int delerr, bool small,
                                              unsigned sact, const float (&sx)[4], unsigned s0, unsigned s1) {
    const int lane = lane_id();
    const unsigned FULL = 0xffffffffu, lt = lanemask_lt();
    const float wsf = pow2f(wse);
    const unsigned im = incon_mask(g);
    const BPh *src = w.bp[w.bpsel];
    BPh *dst = w.bp[w.bpsel ^ 1];
    const int nbp = w.nbp;
    int app = 0;
#pragma unroll 1
    for (int base = 0; base < nbp; base += 32) {
        const int it = base + lane;
        app += __popc(__ballot_sync(FULL, it < nbp && (small ? sact : (unsigned)w.bx[it].act) != 0));
    }
    int k = 0;
#pragma unroll 1
    for (int base = 0; base < nbp; base += 32) {
        const int it = base + lane;
        unsigned act = 0u;
        float x0 = sx[0], x1 = sx[1], x2 = sx[2], x3 = sx[3];
        if (it < nbp) {
            act = sact;
            if (!small) {
                const BXh &x = w.bx[it];
                act = x.act; x0 = x.extp[0]; x1 = x.extp[1]; x2 = x.extp[2]; x3 = x.extp[3];
            }
        }
        const unsigned bs = __ballot_sync(FULL, act != 0);
        const int extra = act ? __popc(act) - 1 : 0;
        // the extensions of the lanes before this one that are appended
        // (at most three each)
        const unsigned e0 = __ballot_sync(FULL, extra & 1), e1 = __ballot_sync(FULL, extra & 2);
        if (act) {
            const BPh b = src[it];
            short2 mm, pm;
            if (small) {   // the positions the new list gives the extensions in s0 / s1
                const unsigned bm = (1u << b.mat) - 1u, bq = (1u << b.pat) - 1u;
                const int n0 = __popc(s0);
                mm = make_short2((short)__popc(s0 & bm), (short)(n0 + __popc(s1 & bm)));
                pm = make_short2((short)__popc(s0 & bq), (short)(n0 + __popc(s1 & bq)));
            } else { mm = w.hapmap[b.mat]; pm = w.hapmap[b.pat]; }
            int pos = app + __popc(e0 & lt) + 2 * __popc(e1 & lt);
            const int own = k + __popc(bs & lt);
#pragma unroll 1
            for (;;) {
                const int ex = top_ext(act);
                act &= ~(1u << ex);
                const int to = act ? pos++ : own;
                const float p = ex == 0 ? x0 : ex == 1 ? x1 : ex == 2 ? x2 : x3;
                if (to < BPMAX) bp_make(dst[to], b, p, ex, ex >> 1 ? mm.y : mm.x, ex & 1 ? pm.y : pm.x, im, wse, wsf, delerr, c.pErr);
                if (!act) break;
            }
        }
        k += __popc(bs);
        app += __popc(e0) + 2 * __popc(e1);
    }
    __syncwarp();
    if (lane == 0) {
        if (app > BPMAX) w.err |= EIMP_ERR_BEAM_CAPACITY;
        w.nbp = min(app, BPMAX);
        w.bpsel ^= 1;
    }
    __syncwarp();
}

// the same for more than 32 beam paths: marks the duplicates, whose table
// entries hold the first path of their key
__device__ __noinline__ bool merge_table(WS &w, const BPh *bp, int n) {
    const int lane = lane_id();
    int2 *ht = reinterpret_cast<int2 *>(w.scr);
    short *slots = reinterpret_cast<short *>(w.scr + 2 * HTS);
    bool anydup = false;
#pragma unroll 1
    for (int i = lane; i < HTS; i += 32) ht[i] = make_int2(-1, INT_MAX);
    __syncwarp();
#pragma unroll 1
    for (int it = lane; it < n; it += 32) {
        const int mr = w.canon[bp[it].mat], pr = w.canon[bp[it].pat];
        const int key = (min(mr, pr) << 16) | max(mr, pr);
        int slot = (int)(((unsigned)key * 2654435761u) >> (32 - HTS_BITS)) & (HTS - 1);
        // linear probing; the table holds at most BPMAX < HTS keys, so a
        // free or matching slot exists within HTS probes
#pragma unroll 1
        for (int probe = 0; probe < HTS; probe++) {
            const int old = atomicCAS(&ht[slot].x, -1, key);
            if (old == -1 || old == key) break;
            slot = (slot + 1) & (HTS - 1);
        }
        atomicMin(&ht[slot].y, it);
        slots[it] = (short)slot;
    }
    __syncwarp();
#pragma unroll 1
    for (int it = lane; it < n; it += 32) {
        const bool dup = ht[slots[it]].y != it;
        w.bx[it].mark = dup ? 1 : -1;
        anydup |= dup;
    }
    return __any_sync(0xffffffffu, anydup);
}

// Beam::mergePaths (Beam.cpp:790-837).  Each beam path's key is the pair of
// first list positions of its two histories (runs of equal histories are
// adjacent in the list).  The first path of each key survives unless a later
// one with the same key is more probable; the duplicates are merged on lane
// 0 in list order (the reference's sequential order within each key), then
// the survivors are compacted into the other buffer.  Up to 32 beam paths
// find their equals by a warp match, more by a hash table.
__device__ __forceinline__ void beam_merge(const Ctx &c, WS &w) {
    const int lane = lane_id();
    const unsigned FULL = 0xffffffffu;
    BPh *bp = w.bp[w.bpsel];
    const int n = w.nbp;
    int2 *ht = reinterpret_cast<int2 *>(w.scr);                    // (key, surviving beam path), x = -1 when free
    short *slots = reinterpret_cast<short *>(w.scr + 2 * HTS);     // table entry of each beam path
    bool anydup = false;
    if (n <= 32) {
        int key = -1 - lane;
        if (lane < n) {
            const int mr = w.canon[bp[lane].mat], pr = w.canon[bp[lane].pat];
            key = (min(mr, pr) << 16) | max(mr, pr);
        }
        const int first = __ffs((int)__match_any_sync(FULL, key)) - 1;
        anydup = __any_sync(FULL, first != lane);
        if (!anydup) return;
        if (lane < n) {
            ht[lane].y = lane;
            slots[lane] = (short)first;
            w.bx[lane].mark = first != lane ? 1 : -1;
        }
    } else anydup = merge_table(w, bp, n);
    __syncwarp();
    if (anydup && lane == 0) {
#pragma unroll 1
        for (int it = 0; it < n; it++) {
            if (w.bx[it].mark != 1) continue;
            BPh &b = bp[it];
            int &rep = ht[slots[it]].y;
            BPh &o = bp[rep];
            if (o.prob > b.prob) {
                o.weight = __fadd_rn(o.weight, __fmul_rn(b.weight, __fdiv_rn(b.prob, o.prob)));
                w.bx[it].mark = -2;
            } else {
                b.weight = __fadd_rn(b.weight, __fmul_rn(o.weight, __fdiv_rn(o.prob, b.prob)));
                w.bx[rep].mark = -2;
                w.bx[it].mark = -1;
                rep = it;
            }
        }
    }
    __syncwarp();
    if (anydup) {
        BPh *dst = w.bp[w.bpsel ^ 1];
        int keep = 0;
#pragma unroll 1
        for (int base = 0; base < n; base += 32) {
            const int it = base + lane;
            const bool alive = it < n && w.bx[it].mark != -2;
            const unsigned ba = __ballot_sync(FULL, alive);
            if (alive) dst[keep + __popc(ba & lanemask_lt())] = bp[it];
            keep += __popc(ba);
        }
        __syncwarp();
        if (lane == 0) { w.nbp = keep; w.bpsel ^= 1; }
    }
    __syncwarp();
}

// Beam::advanceBeamFront (Beam.cpp:263-539)
__device__ __forceinline__ int beam_advance(const Ctx &c, WS &w, int &ncmd) {
    const int lane = lane_id();
    // every lane has read the cursor for its loop condition before lane 0
    // moves it (otherwise lanes could leave the caller's loop at different
    // iterations and meet different warp collectives)
    __syncwarp();
    const int cursor = w.cursor + (w.reverse ? -1 : 1), nbp = w.nbp, nhap = w.nhap;
    const bool small = nbp <= 32 && nhap <= 32;
    const BPh *bp = w.bp[w.bpsel];
    Cons cn;
    cn.type = w.reverse && cursor == c.S - 1 ? C_HETKEEP : C_NONE;   // (Target.cpp:650)
    cn.refidx = 0;
    if (w.constr) cn = w.constr[cursor];
    const int g = c.tg[cursor];
    __syncwarp();
    if (lane == 0) { w.cursor = cursor; w.step++; }
    __syncwarp();
    if (c.warps == 1) beam_next(c, w, w.step);
    float x[4] = {0.0f, 0.0f, 0.0f, 0.0f};
    unsigned act = 0u;
    int wse = 0, delerr = 0;
    bool regs;   // the surviving extensions are in x / act, of the haplotype paths in s0 / s1
    unsigned s0 = 0u, s1 = 0u;
    while (true) {
        // markRequiredExtensions (only sets flags: order free)
        unsigned m0 = 0u, m1 = 0u;
        if (small) {
            if (lane < nbp) {
                const int mat = bp[lane].mat, pat = bp[lane].pat;
                int rm = 3, rp = 3;
                if (cn.type != C_NONE) {
                    rm = hp_required(c.hp(w.happ[mat]), cn);
                    rp = hp_required(c.hp(w.happ[pat]), cn);
                }
                m0 = (unsigned)(rm & 1) << mat | (unsigned)(rp & 1) << pat;
                m1 = (unsigned)(rm >> 1) << mat | (unsigned)(rp >> 1) << pat;
            }
            m0 = warp_or(m0);
            m1 = warp_or(m1);
            if (lane < nhap) {
                w.tox[0][lane] = (unsigned char)((m0 >> lane) & 1u);
                w.tox[1][lane] = (unsigned char)((m1 >> lane) & 1u);
            }
        } else {
#pragma unroll 1
            for (int i = lane; i < nhap; i += 32) { w.tox[0][i] = 0; w.tox[1][i] = 0; }
            __syncwarp();
#pragma unroll 1
            for (int q = lane; q < 2 * nbp; q += 32) {
                const int pos = q & 1 ? bp[q >> 1].pat : bp[q >> 1].mat;
                const int r = hp_required(c.hp(w.happ[pos]), cn);
                if (r & 1) w.tox[0][pos] = 1;
                if (r & 2) w.tox[1][pos] = 1;
            }
        }
        // haplotype-path extensions
        beam_command(c, w, ncmd, CMD_WALK);
        beam_walk(c, w);
        if (c.warps > 1) block_barrier(32 * c.warps);
        int minse = 0, maxse = INT_MIN;
#pragma unroll 1
        for (int i = lane; i < nhap; i += 32)
            if (w.tox[0][i] | w.tox[1][i]) { minse = min(minse, w.ese[i]); maxse = max(maxse, w.ese[i]); }
        minse = warp_mini(minse);
        maxse = warp_maxi(maxse);
        const int bpscaleexp = -(maxse + minse);
        // beam-path extensions and pruning
        int ok = -1;
        regs = small;
        if (small) {
            float mp = 0.0f, weight = 1.0f;
            int nErr = 0;
            act = 0u;
            if (lane < nbp) {
                const BPh &b = bp[lane];
                weight = b.weight;
                nErr = b.nErr;
                act = bp_extend(c, w, b, g, cn, bpscaleexp, x);
#pragma unroll
                for (int ex = 0; ex < 4; ex++)
                    if (((act >> ex) & 1u) && mp < x[ex]) mp = x[ex];
            }
            mp = warp_maxf(mp);
            const unsigned cand = act;
            ok = prune_small(w, __fmul_rn(c.pLimit, mp), weight, nErr, x, act, wse, delerr);
            if (ok > 0) {
                // a haplotype-path extension stays active while a surviving
                // beam path uses it, or when none used it (constraints only)
                int mat = 0, pat = 0;
                if (lane < nbp) { mat = bp[lane].mat; pat = bp[lane].pat; }
                s0 = warp_or((act & 3u ? 1u << mat : 0u) | (act & 5u ? 1u << pat : 0u));
                s1 = warp_or((act & 12u ? 1u << mat : 0u) | (act & 10u ? 1u << pat : 0u));
                if (cn.type != C_NONE) {
                    s0 |= m0 & ~warp_or((cand & 3u ? 1u << mat : 0u) | (cand & 5u ? 1u << pat : 0u));
                    s1 |= m1 & ~warp_or((cand & 12u ? 1u << mat : 0u) | (cand & 10u ? 1u << pat : 0u));
                }
                if (lane < nhap) w.hact[lane] = (unsigned char)(((s0 >> lane) & 1u) | ((s1 >> lane) & 1u) << 1);
                __syncwarp();
            }
        }
        if (ok < 0) {
            regs = false;
            const float maxP = extend_general(c, w, cn, g, bpscaleexp);
            ok = beam_prune_select(w, c.pLimit, maxP, cn.type == C_NONE);
            wse = w.wse;
            delerr = w.delerr;
        }
        if (c.warps > 2) {
            if (lane == 0) w.ires = ok;
            pair_barrier(1, 64);
        }
        if (ok) break;
        if (cn.type != C_NONE) { cn.type = C_NONE; continue; }
        if (lane == 0) w.err |= EIMP_ERR_BEAM_EMPTY;
        __syncwarp();
        return -1;
    }
    const bool apart = c.warps > 2;
    if (!apart) {
        beam_apply_hap(c, w);
        if (w.err) return -1;
        beam_canon(c, w);
        beam_copy(c, w, 0, 1);
        __syncwarp();
    } else if (!regs) pair_barrier(2, 64);   // the new list positions
    beam_apply_bp(c, w, g, wse, delerr, regs, act, x, s0, s1);
    if (apart && regs) pair_barrier(2, 64);
    if (w.err) return -1;
    beam_merge(c, w);
    return 0;
}

// Beam::callKeepPhaseProb (Beam.cpp:95-185) for call ci, against the call
// before it or (twoback) the one before that, and Beam::callDosage
// (Beam.cpp:187-261) for split site ds when ci < 0: the beam advances to the
// call's front, the lanes classify the beam paths and prepare each path's
// terms of the two sums (0 where a path adds nothing, which leaves a float
// sum unchanged), lane 0 adds them in list order.  One function with one copy
// of the advance: its code has to stay in the SM's instruction cache.
__device__ __forceinline__ float beam_call(const Ctx &c, WS &w, int &ncmd, int ci, bool twoback, int ds) {
    const int lane = lane_id();
    const bool keep = ci >= 0, rev = w.reverse != 0;
    const int cl = keep ? c.calls[ci] : ds;
    const int front = rev ? max(cl - w.Delta, 0) : min(cl + w.Delta, c.S - 1);
    const int curridx = rev ? cl - front : front - cl;
    int refidx = -1;
    if (keep) {
        const int r = c.calls[ci + (rev ? 1 : -1) * (twoback ? 2 : 1)];
        refidx = rev ? r - front : front - r;
    }
    while (rev ? w.cursor > front : w.cursor < front)
        if (beam_advance(c, w, ncmd)) return -1.0f;
    const BPh *bp = w.bp[w.bpsel];
    const int n = w.nbp;
#pragma unroll 1
    for (int it = lane; it < n; it += 32) {
        const BPh &b = bp[it];
        const HPh &hm = c.hp(w.happ[b.mat]), &hq = c.hp(w.happ[b.pat]);
        const int cf = bh_at(hm, curridx), cs = bh_at(hq, curridx);
        const float p = __fmul_rn(b.weight, b.prob);
        float k, s;
        if (keep) {
            const int rf = bh_at(hm, refidx), rs = bh_at(hq, refidx);
            if (cf != cs && rf != rs) {
                k = cf == rf ? p : 0.0f;
                s = cf == rf ? 0.0f : p;
            } else {
                k = __fdiv_rn(p, 2.0f);
                s = k;
            }
        } else {
            k = cf == cs ? (cf == 1 ? __fmul_rn(2.0f, p) : 0.0f) : p;
            s = p;
        }
        w.scr[it] = k; w.scr[BPMAX + it] = s;
    }
    __syncwarp();
    // every lane adds the same values in the same order
    float acck = 0.0f, accs = 0.0f;
#pragma unroll 4
    for (int it = 0; it < n; it++) { acck = __fadd_rn(acck, w.scr[it]); accs = __fadd_rn(accs, w.scr[BPMAX + it]); }
    __syncwarp();
    if (keep) {
        const float t = __fadd_rn(acck, accs);
        return t > 0.0f ? __fdiv_rn(acck, t) : 0.5f;
    }
    return accs > 0.0f ? __fdiv_rn(acck, accs) : 1.0f;
}

__host__ __device__ __forceinline__ size_t align256(size_t x) { return (x + 255) & ~(size_t)255; }

}  // namespace


// arena layout per target (bytes)
struct ArenaLayout {
    size_t hp, ph, ivpool, cd, heap, cons, rcons, probs, confs, tg, total;
    int NH, HMAX;
    int NS;   // haplotype-path slots in shared memory (set by the launcher)
    int NR;   // of which and of more the records
};

static ArenaLayout arena_layout(const BeamParams &p, int M) {
    ArenaLayout a;
    int P = p.P > p.Pf ? p.P : p.Pf;
    int H = p.H > p.Hf ? p.H : p.Hf;
    a.NH = 4 * P + 8;
    a.HMAX = H;
    a.NS = 0;
    a.NR = 0;
    size_t o = 0;
    a.hp = o; o = align256(o + sizeof(HPh) * a.NH);
    a.ph = o; o = align256(o + sizeof(float) * PHMAX * a.NH);
    // the interval pool doubles as the storage of the pre-phasing constraint
    // heaps (one entry per split site) once the fast beam is done
    const size_t ivb = sizeof(uint32_t) * (size_t)H * 3 * a.NH, heapb = sizeof(Hel) * (size_t)(M + 1);
    a.ivpool = o; o = align256(o + (ivb > heapb ? ivb : heapb));
    a.cd = o; o = align256(o + sizeof(float) * 32 * (size_t)H);
    a.heap = o; o = align256(o + sizeof(Hel) * (PMAX + 2));
    a.cons = o; o = align256(o + sizeof(Cons) * (size_t)(M + 1));
    a.rcons = o; o = align256(o + sizeof(Cons) * (size_t)(M + 1));
    a.probs = o; o = align256(o + sizeof(float) * (size_t)(M + 1));
    a.confs = o; o = align256(o + sizeof(float) * (size_t)(M + 1));
    a.tg = o; o = align256(o + (size_t)(M + 1));
    a.total = o;
    return a;
}

size_t beam_arena_bytes(const BeamParams &p, int M) { return arena_layout(p, M).total; }

// shared memory of a target besides its WS: the ring of PBWT row pairs (three, or
// two where a pair takes more than 8 KB), the merge key of each haplotype
// path, and the haplotype-path slots
__host__ __device__ __forceinline__ int beam_ring(int K) { return K <= 16384 ? 3 : 2; }
__host__ __device__ __forceinline__ size_t beam_rows_bytes(int K) { return (size_t)beam_ring(K) * 2 * eimp_kw(K) * 4; }
__host__ __device__ __forceinline__ size_t beam_canon_bytes(int NH) { return (((size_t)NH * 2 + 15) / 16) * 16; }
// strides of a slot: the ring (a power of two >= H, at least 4) and the
// interval buffers (odd, so that the paths' lanes hit different banks)
__host__ __device__ __forceinline__ int slot_ring(int H) { int n = 4; while (n < H) n <<= 1; return n; }
__host__ __device__ __forceinline__ int slot_buf(int H) { return H | 1; }
__host__ __device__ __forceinline__ size_t beam_term_bytes(int warps) { return (size_t)(warps - 1) * 2 * WITEMS * sizeof(float); }
__host__ __device__ __forceinline__ size_t beam_slot_bytes(int NS, int H, int NR) {
    return (sizeof(HPh) * NR + (4 * (size_t)slot_ring(H) + 12 * (size_t)slot_buf(H)) * NS + 15) / 16 * 16;
}

// a bit of a row of words set or cleared, without waiting for the word
__device__ __forceinline__ void setbit_(uint64_t *v, int i) {
    atomicOr(reinterpret_cast<unsigned long long *>(v) + (i >> 6), 1ull << (i & 63));
}
__device__ __forceinline__ void clrbit_(uint64_t *v, int i) {
    atomicAnd(reinterpret_cast<unsigned long long *>(v) + (i >> 6), ~(1ull << (i & 63)));
}

// Targets in longest-first order: order[rank] = target, ranked by split sites
// descending, ties by index.  One CTA; the persistent beam below takes the
// targets in this order, so the longest walks start first and the short ones
// fill the end of the launch.
__global__ void lpt_order_kernel(const int32_t *__restrict__ nsplits, int ntgt, int32_t *__restrict__ order,
                                 const int *__restrict__ skip) {
    if (skip && *skip) return;
    for (int i = threadIdx.x; i < ntgt; i += blockDim.x) {
        const int si = nsplits[i];
        int rank = 0;
        for (int j = 0; j < ntgt; j++) {
            const int sj = nsplits[j];
            rank += sj > si || (sj == si && j < i);
        }
        order[rank] = i;
    }
}

// The constraints kept from the pre-phasing pass (Target.cpp:402-436); lane 0.
__device__ __noinline__ void constraint_heaps(Hel *hq, Cons *cons, const float *phaseProbs, const int32_t *calls, int S,
                                              float minfixsize, float maxfixsize, float minfixthr, float maxfixthr) {
    // the constraint heaps (Target.cpp:402-436), filled in site order as
    // the reference does; the interval pool of the finished fast beam
    // serves as heap storage
    for (int pass = 0; pass < 2; pass++) {   // 0: call sites, 1: homozygous split sites
        int n = 0;
        int nci2 = 1;
        for (int si = 1; si < S; si++) {
            bool iscall = (si == calls[nci2]);
            if (iscall) nci2++;
            if ((pass == 0) == iscall) heap_push(hq, n, phaseProbs[si], si, 0);
        }
        const size_t total = (size_t)n;
        const size_t smin = (size_t)__fmul_rn((float)total, minfixsize);
        const size_t smax = (size_t)((double)total * (1.0 - (double)maxfixsize));
        size_t si;
        const double thrmax = pass == 0 ? (double)maxfixthr - 0.5 : (double)maxfixthr * 2.0;
        const double thrmin = pass == 0 ? (double)minfixthr - 0.5 : (double)minfixthr * 2.0;
        for (si = 0; si < smin; si++) {
            Hel cc = heap_popmin(hq, n);
            if ((double)cc.key >= thrmax || ((double)cc.key >= thrmin && si >= smax)) break;
            cons[cc.a].type = C_NONE;
        }
        if (pass == 0 && si == smin) {
            // (Target.cpp:416-425: compared against the shrinking heap)
            for (; si < (size_t)n; si++) {
                Hel cc = heap_popmin(hq, n);
                if (cc.key > 0.0f) break;
                cons[cc.a].type = C_NONE;
            }
        }
    }
}

// Target::phaseExtPBWT (Target.cpp:291-777), one CTA per target.  The grid
// is persistent (as many CTAs as are resident at once): every CTA takes the
// next target from a device counter, in the order given (longest first), and
// phases it with its own beam arena, so the arenas number the resident CTAs,
// not the targets.
__device__ __forceinline__ void beam_run(
    const BeamParams &p, const ArenaLayout &al, int ntgt, int M, const uint8_t *__restrict__ gt, const uint64_t *__restrict__ monos,
    const int32_t *__restrict__ splits, const int32_t *__restrict__ nsplits, const int32_t *__restrict__ calls,
    const int32_t *__restrict__ ncalls, const float *__restrict__ cmdiffs, const uint32_t *__restrict__ pbwt,
    const int32_t *__restrict__ count0, const int64_t *__restrict__ rowoff, uint8_t *__restrict__ arena,
    size_t arena_bytes, uint64_t *__restrict__ mats, uint64_t *__restrict__ pats, float *__restrict__ dmat,
    float *__restrict__ dpat, float *__restrict__ totalconf, int32_t *__restrict__ ncallsites,
    uint32_t *__restrict__ status, const int *__restrict__ skip, const int32_t *__restrict__ order,
    int *__restrict__ workq) {
    if (skip && *skip) return;   // the batch exceeds the reserved rows
    extern __shared__ __align__(16) uint8_t smem_raw[];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, warps = blockDim.x >> 5;
    WS &w = *reinterpret_cast<WS *>(smem_raw);
    uint8_t *const ab = arena + (size_t)blockIdx.x * arena_bytes;
    int ncmd = 0;   // commands given for the current target
    for (;;) {
    int qi = 0;
    if (wid == 0 && lane == 0) w.qi = qi = atomicAdd(workq, 1);
    if (warps > 1) { block_barrier(32 * warps); qi = w.qi; }
    else qi = __shfl_sync(0xffffffffu, qi, 0);
    if (qi >= ntgt) break;
    const int t = order[qi];
    const int wM = (int)eimp_W(M);
    const uint8_t *g = gt + (size_t)t * M;
    const uint64_t *mo = monos + (size_t)t * wM;
    uint64_t *mat = mats + (size_t)t * wM;
    uint64_t *pat = pats + (size_t)t * wM;
    float *dm = dmat + (size_t)t * M;
    float *dp = dpat + (size_t)t * M;
    const int S = nsplits[t];
    const int C = ncalls[t];
    const int K = p.K;
    const size_t kw = eimp_kw(K);
    // after the WS: the ring, the merge keys, the slots, the other warps' walk terms
    uint8_t *const ring = smem_raw + sizeof(WS);
    uint8_t *const canon = ring + beam_rows_bytes(K);
    uint8_t *const slots = canon + beam_canon_bytes(al.NH);
    Ctx c;
    c.wid = wid; c.warps = warps;
    c.term = wid ? reinterpret_cast<float *>(slots + beam_slot_bytes(al.NS, al.HMAX, al.NR)) + (wid - 1) * 2 * WITEMS : w.scr;
    c.NS = al.NS; c.NR = al.NR; c.NH = al.NH;
    c.HS = slot_buf(al.HMAX); c.HG = al.HMAX; c.PHS = slot_ring(al.HMAX);
    c.phs = reinterpret_cast<float *>(slots);
    c.hps = reinterpret_cast<HPh *>(c.phs + (size_t)al.NS * c.PHS);
    c.ivs = reinterpret_cast<uint32_t *>(c.hps + al.NR);
    c.hpg = reinterpret_cast<HPh *>(ab + al.hp);
    c.phg = reinterpret_cast<float *>(ab + al.ph);
    c.ivg = reinterpret_cast<uint32_t *>(ab + al.ivpool);
    c.cdb = reinterpret_cast<float *>(ab + al.cd);
    c.ring = reinterpret_cast<uint32_t *>(ring);
    c.nring = beam_ring(K);
    Cons *cons = reinterpret_cast<Cons *>(ab + al.cons);
    Cons *rcons = reinterpret_cast<Cons *>(ab + al.rcons);
    float *phaseProbs = reinterpret_cast<float *>(ab + al.probs);
    float *callConfs = reinterpret_cast<float *>(ab + al.confs);
    uint8_t *tg = ab + al.tg;
    const int64_t r0 = rowoff[t];
    c.Mp = 2 * S + 1;
    c.rows = pbwt + (size_t)2 * r0 * kw;
    c.K = K; c.kw = (int)kw;
    c.Kinv = (float)(1.0 / (double)(float)K);
    c.cmd = cmdiffs + (size_t)t * (M + 1);
    c.S = S;
    c.calls = calls + (size_t)t * M;
    c.tg = tg;
    c.pErr = p.pErr; c.pLimit = p.pLimit; c.expectIBDcM = p.expectIBDcM;
    const int32_t *sp = splits + (size_t)t * M;
    if (wid) {   // the first warp runs the beam, the others help
        beam_help(c, w);
        continue;
    }
    ncmd = 0;
    for (int i = lane; i < wM; i += 32) { mat[i] = 0ull; pat[i] = 0ull; }
    for (int i = lane; i < M; i += 32) { dm[i] = 0.0f; dp[i] = 0.0f; }
    for (int s = lane; s < S; s += 32) {
        tg[s] = g[sp[s]];
        if (p.doPrePhasing) { cons[s].type = C_NONE; cons[s].refidx = 0; }
    }
    if (lane == 0) {
        w.canon = reinterpret_cast<short *>(canon);
        w.heap = reinterpret_cast<Hel *>(ab + al.heap);
    }
    __syncwarp();

    int err = 0;
    const int startph = p.startph ? (p.startph[t] != 0) : 0;   // VCFData::getStartPhase (Target.cpp:311-312)
    const int stop = S > 0 ? sp[c.calls[0]] : M;               // the first call site
    int cur = startph, lastph = startph;
    int nprobs = 0;
    // pass 0: pre-phasing (Target.cpp:324-438); 1: fine phasing forward
    // (:458-599); 2: backward (:620-758).  One loop over the passes' calls.
    for (int pass = p.doPrePhasing ? 0 : 1; pass < 3 && !err; pass++) {
        if (pass == 0) {
            if (lane == 0 && S > 0) { cons[0].type = C_HETKEEP; cons[0].refidx = 0; }
        } else if (pass == 1) {
            cur = startph;   // Target.cpp:443
            if (lane == 0) phaseProbs[0] = 0.0f;
            nprobs = 1;
        } else {
            if (S == 0) break;
            // Target.cpp:601-619
            for (int i = lane; i < C; i += 32) callConfs[i] = 0.0f;
            __syncwarp();
            if (lane == 0) {
                if (p.doRevPhasing) callConfs[C - 1] = (float)((double)fabsf(phaseProbs[nprobs - 1]) + 0.5);
                else for (int i = 0; i < nprobs && i < C; i++) callConfs[i] = (float)((double)fabsf(phaseProbs[i]) + 0.5);
            }
            __syncwarp();
            if (!p.doRevPhasing) break;
            for (int s = lane; p.doPrePhasing && s < S; s += 32) { rcons[s].type = C_NONE; rcons[s].refidx = 0; }
            __syncwarp();
            if (lane == 0) {
                for (int ci = 1; p.doPrePhasing && ci < S; ci++) {
                    Cons cc = cons[ci];
                    if (cc.type == C_HETKEEP || cc.type == C_HETSWITCH) {
                        Cons &r = rcons[ci - cc.refidx - 1];
                        if (r.type != C_NONE) {
                            int ridx = ci - cc.refidx + r.refidx;
                            rcons[ridx].refidx = cc.refidx - r.refidx - 1;
                            rcons[ridx].type = (cc.type != r.type) ? C_HETSWITCH : C_HETKEEP;
                        } else { r.type = cc.type; r.refidx = cc.refidx; }
                    } else if (cc.type == C_HOMREF || cc.type == C_HOMALT) {
                        rcons[ci].type = cc.type;
                    }
                }
                if (p.doPrePhasing) { rcons[S - 1].type = C_HETKEEP; rcons[S - 1].refidx = 0; }
                float last = phaseProbs[nprobs - 1];
                float dref = last < 0.0f ? (float)(0.5 + (double)last) : (float)(0.5 - (double)last);
                float dalt = last < 0.0f ? (float)(0.5 - (double)last) : (float)(0.5 + (double)last);
                int site = sp[c.calls[C - 1]];
                dm[site] = cur == 0 ? dref : dalt;
                dp[site] = cur == 0 ? dalt : dref;
            }
        }
        __syncwarp();
        beam_init(c, w, p.doPrePhasing ? (pass == 2 ? rcons : cons) : nullptr, pass == 2, pass ? p.H : p.Hf, pass ? p.P : p.Pf, pass ? p.Delta : p.Deltaf);
        beam_command(c, w, ncmd, CMD_NEXT);
        int nci = 1, si = 1, rci = C - 2;   // the next call of pass 0 and 1, split site of pass 0, call of pass 2
        bool second = false;                // pass 0: the call against the one two back follows
        float prone = 0.0f;
        // pass 1, 32 sites at a time: the homozygous sites and the
        // heterozygous ones without a call are set by the lanes, the calls
        // follow one another
        int b = -32, gg = 3;
        unsigned het = 0u, mono = 0u, mw = 0u, pw = 0u;
        for (;;) {
            int ci = -1, ds = -1;
            if (pass == 0) {
                if (si >= S) break;
                if (si == c.calls[nci]) ci = nci;
                else ds = si;
            } else if (pass == 1) {
                for (;;) {
                    for (; het; het &= het - 1) {
                        const int j = __ffs((int)het) - 1;
                        if (b + j > stop && !((mono >> j) & 1u)) { ci = nci; break; }
                        if (b + j >= stop && cur) mw |= 1u << j;
                        else pw |= 1u << j;
                    }
                    if (ci >= 0) break;
                    if (b >= 0 && lane == 0) {
                        reinterpret_cast<uint32_t *>(mat)[b >> 5] = mw;
                        reinterpret_cast<uint32_t *>(pat)[b >> 5] = pw;
                    }
                    b += 32;
                    if (b >= M) break;
                    const int m = b + lane;
                    gg = m < M ? g[m] : 3;
                    mono = reinterpret_cast<const uint32_t *>(mo)[b >> 5];
                    mw = pw = __ballot_sync(0xffffffffu, gg == 2);
                    het = __ballot_sync(0xffffffffu, gg == 1);
                    if (gg == 2) { dm[m] = 1.0f; dp[m] = 1.0f; }
                    else if (gg == 1 && (m < stop || (m > stop && ((mono >> lane) & 1u)))) { dm[m] = 0.5f; dp[m] = 0.5f; }
                }
                if (ci < 0) break;
            } else {
                if (rci < 0) break;
                ci = rci;
            }
            float pr = beam_call(c, w, ncmd, ci, second, ds);
            if (w.err) { err = 1; break; }
            if (ci >= 0) pr = (float)((double)pr - 0.5);
            if (pass == 0) {
                if (ci >= 0) {
                    if (nci > 1 && !second) { second = true; prone = pr; continue; }
                    int ref = cur, refidx = c.calls[nci] - c.calls[nci - 1] - 1;
                    if (second) {
                        const float p2 = pr;
                        pr = prone;
                        if (fabsf(p2) > fabsf(pr)) { pr = p2; ref = lastph; refidx = c.calls[nci] - c.calls[nci - 2] - 1; }
                        second = false;
                    }
                    lastph = cur;
                    int type;
                    if (pr < 0.0f) { cur = !ref; type = C_HETSWITCH; } else { cur = ref; type = C_HETKEEP; }
                    if (lane == 0) { cons[si].type = type; cons[si].refidx = refidx; phaseProbs[si] = fabsf(pr); }
                    nci++;
                } else if (lane == 0) {
                    cons[si].refidx = 0;
                    if (tg[si] == 0) { cons[si].type = C_HOMREF; pr = (float)(2.0 - (double)pr); }
                    else cons[si].type = C_HOMALT;
                    phaseProbs[si] = pr;
                }
                si++;
                __syncwarp();
            } else if (pass == 1) {
                if (lane == 0) phaseProbs[nprobs] = pr;
                nprobs++;
                cur = pr < 0.0f ? !cur : cur;
                nci++;
                const unsigned bit = het & (0u - het);
                if (cur) mw |= bit;
                else pw |= bit;
                het &= het - 1;
            } else {
                float fw = phaseProbs[rci + 1];
                if (fabsf(fw) > fabsf(pr)) pr = fw;
                cur = pr < 0.0f ? !cur : cur;
                if (lane == 0) {
                    int s2 = sp[c.calls[rci]];
                    if (cur) { setbit_(mat, s2); clrbit_(pat, s2); } else { clrbit_(mat, s2); setbit_(pat, s2); }
                    float dref = pr < 0.0f ? (float)(0.5 + (double)pr) : (float)(0.5 - (double)pr);
                    float dalt = pr < 0.0f ? (float)(0.5 - (double)pr) : (float)(0.5 + (double)pr);
                    dm[s2] = cur == 0 ? dref : dalt;
                    dp[s2] = cur == 0 ? dalt : dref;
                    callConfs[rci] = (float)((double)fabsf(pr) + 0.5);
                }
                __syncwarp();
                rci--;
            }
        }
        // the other warps are done with the pass: the copies of the paths that
        // split last write the interval pool, the heaps' storage, and the next
        // pass starts with new paths in it
        beam_command(c, w, ncmd, CMD_MEET);
        if (pass == 0 && !err && lane == 0)
            constraint_heaps(reinterpret_cast<Hel *>(c.ivg), cons, phaseProbs, c.calls, S, p.minfixsize, p.maxfixsize,
                             p.minfixthr, p.maxfixthr);
        __syncwarp();
    }
    if (lane == 0) {
        float tc = 0.0f;
        int nc = 0;
        if (!err && S > 0) {   // Target.cpp:761-772
            for (int i = 0; i < C; i++) tc = __fadd_rn(tc, callConfs[i]);
            nc = C;
        }
        totalconf[t] = tc;
        ncallsites[t] = nc;
        if (err) atomicOr(status, w.err ? w.err : (uint32_t)EIMP_ERR_BEAM_EMPTY);
    }
    beam_command(c, w, ncmd, CMD_EXIT);
    __syncwarp();
    }
    copy_async_wait<0>();
}

__global__ void __launch_bounds__(BEAM_SM_CTAS * 32 * BEAM_WARPS, 1) beam_kernel(
    BeamParams p, ArenaLayout al, int ntgt, int M, const uint8_t *__restrict__ gt, const uint64_t *__restrict__ monos,
    const int32_t *__restrict__ splits, const int32_t *__restrict__ nsplits, const int32_t *__restrict__ calls,
    const int32_t *__restrict__ ncalls, const float *__restrict__ cmdiffs, const uint32_t *__restrict__ pbwt,
    const int32_t *__restrict__ count0, const int64_t *__restrict__ rowoff, uint8_t *__restrict__ arena,
    size_t arena_bytes, uint64_t *__restrict__ mats, uint64_t *__restrict__ pats, float *__restrict__ dmat,
    float *__restrict__ dpat, float *__restrict__ totalconf, int32_t *__restrict__ ncallsites,
    uint32_t *__restrict__ status, const int *__restrict__ skip, const int32_t *__restrict__ order,
    int *__restrict__ workq) {
    beam_run(p, al, ntgt, M, gt, monos, splits, nsplits, calls, ncalls, cmdiffs, pbwt, count0, rowoff, arena, arena_bytes, mats,
                      pats, dmat, dpat, totalconf, ncallsites, status, skip, order, workq);
}

// The launch: with a target or less per SM, one CTA of BEAM_MAX_WARPS warps on
// each; with more, CTAs of BEAM_WARPS warps, as many per SM as the targets fill, at
// most BEAM_SM_CTAS.  The shared memory that is left becomes haplotype-path slots:
// all of it with a target or less per SM, a BEAM_SM_CTAS-th with more -- a second
// context's beams then find room beside the last targets of the first (192
// targets of 32,000 sites, three contexts in turn: 57.5 -> 45.5 ms a pass; the
// price is a single context's pass, 61.8 -> 63.0 ms), and slots that go to the
// arena for it cost little (1,000 targets of 5,000 sites, one CTA per SM: 107 ms
// with all slots in shared memory, 112 with 12).
struct BeamShape { int warps, ctas; size_t smem; };

static size_t beam_smem(const BeamParams &p, const ArenaLayout &al, int warps) {
    return sizeof(WS) + beam_rows_bytes(p.K) + beam_canon_bytes(al.NH) + beam_slot_bytes(al.NS, al.HMAX, al.NR) +
           beam_term_bytes(warps);
}

static bool beam_shape(const BeamParams &p, ArenaLayout &al, int ntgt, BeamShape &s, int *sms) {
    int dev = 0, nsm = 0, lim = 0, sm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&lim, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) != cudaSuccess)
        return false;
    *sms = nsm;
    int per = (ntgt + nsm - 1) / nsm;   // CTAs on an SM
    s.warps = per > 1 ? BEAM_WARPS : BEAM_MAX_WARPS;
    if (per > BEAM_SM_CTAS) per = BEAM_SM_CTAS;
    al.NS = 0;
    const size_t base = beam_smem(p, al, s.warps);
    if (base > (size_t)lim) return false;
    size_t room;   // of each CTA, 1 KB of it the system's
    for (;; per--) {
        room = (size_t)sm / (per > 1 ? BEAM_SM_CTAS : 1) - 1024;
        if (room < base) room = (size_t)sm / per - 1024;
        if (room > (size_t)lim) room = (size_t)lim;
        if (per == 1 || base <= room) break;
    }
    // records first (40 bytes each, for a beam of a usual size), then slots
    al.NR = al.NH < BEAM_RECORDS ? al.NH : BEAM_RECORDS;
    while (al.NR > 0 && beam_smem(p, al, s.warps) > room) al.NR -= al.NR < 8 ? 1 : 8;
    const size_t one = beam_slot_bytes(16, al.HMAX, 0) / 16, used = beam_smem(p, al, s.warps);
    al.NS = used < room ? (int)((room - used) / one) : 0;
    if (al.NS > al.NR) al.NS = al.NR;
    while (al.NS > 0 && beam_smem(p, al, s.warps) > room) al.NS--;
    s.smem = beam_smem(p, al, s.warps);
    s.ctas = ntgt < per * nsm ? ntgt : per * nsm;
    return true;
}

int beam_slots(const BeamParams &p, int M, int ntgt, int pct) {
    ArenaLayout al = arena_layout(p, M);
    BeamShape s;
    int nsm = 0;
    if (!beam_shape(p, al, ntgt, s, &nsm)) return -1;
    const int part = (int)((long)s.ctas * (pct < 1 ? 1 : pct > 100 ? 100 : pct) / 100);
    return part < 1 ? 1 : part;
}

cudaError_t launch_beam(const BeamParams &p, int ntgt, int M, const uint8_t *gt, const uint64_t *monos,
                        const int32_t *splits, const int32_t *nsplits, const int32_t *calls, const int32_t *ncalls,
                        const float *cmdiffs, const uint32_t *pbwt, const int32_t *count0, const int64_t *rowoff,
                        void *arena, size_t arena_bytes, int slots, int32_t *order, int *workq, uint64_t *mats,
                        uint64_t *pats, float *dmat, float *dpat, float *totalconf, int32_t *ncallsites,
                        uint32_t *status, const int *skip, cudaStream_t st) {
    ArenaLayout al = arena_layout(p, M);
    BeamShape s;
    int nsm = 0;
    if (!beam_shape(p, al, ntgt, s, &nsm)) return cudaErrorInvalidValue;
    if (arena_bytes < al.total || slots < 1) return cudaErrorInvalidValue;
    cudaError_t e = ensure_dynamic_smem((const void *)beam_kernel, s.smem);
    if (e != cudaSuccess) return e;
    lpt_order_kernel<<<1, 1024, 0, st>>>(nsplits, ntgt, order, skip);
    if ((e = launched()) != cudaSuccess) return e;
    if ((e = cudaMemsetAsync(workq, 0, sizeof(int), st)) != cudaSuccess) return e;
    beam_kernel<<<slots, 32 * s.warps, s.smem, st>>>(p, al, ntgt, M, gt, monos, splits, nsplits, calls,
                                                              ncalls, cmdiffs, pbwt, count0, rowoff,
                                                              (uint8_t *)arena, arena_bytes, mats, pats, dmat, dpat,
                                                              totalconf, ncallsites, status, skip, order, workq);
    return launched();
}

}  // namespace eimp
