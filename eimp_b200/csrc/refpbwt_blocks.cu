// Checkpoint orders of the reference PBWT by blocks of sites, for B200
// (sm_100a).
//
// The order before site m + n is the order before site m stably sorted by the
// haplotypes' alleles at sites m .. m + n - 1, the last site most significant
// (PBWT.cpp:207-285 one site at a time).  Of a block of sites only the ranking
// of its allele patterns matters, and that is the same whatever the order
// before it: so
//  * launch_block_keys (a transpose, imp_kernels.cu) gives every haplotype its 64
//                     alleles of a block as one number, the last site its
//                     highest bit;
//  * rp_class_kernel  replaces them by their dense rank, a CTA per block: the
//                     haplotypes of a block share few patterns, so a rank has
//                     ten bits or so instead of 64.  A second launch
//                     ranks groups of consecutive blocks by their blocks'
//                     ranks;
//  * rp_order_kernel  walks the groups one after the other, sorting the order by
//                     each group's ranks (one CTA, the only serial part), then
//                     in a second launch the blocks of every group, a CTA per
//                     group from the order before it;
//  * rw_count_kernel, rw_place_kernel   sort by one block's ranks after another
//                     with the whole GPU where the orders outgrow an SM's
//                     shared memory;
//  * rp_sub_kernel (or the same passes over all blocks at once) adds the orders
//                     every RB_SUB sites inside the blocks, from which
//                     refpbwt_fill_sub_kernel's CTAs write the rest.
// With the group size near the square root of the number of blocks the serial
// chain is two square roots of it long, a few counting-sort passes each, instead
// of 13 passes per block (refpbwt_ckpt_kernel).
//
// Scratch: a block's numbers, ranks and orders live in the prefix arrays of
// its own later sites, which the fill pass writes afterwards.
#include <climits>

#include "common.cuh"
#include "kernels.h"

namespace eimp {

constexpr int RB_SITES = REFPBWT_BLOCK;   // sites of a block
constexpr int RB_BITS = 20;     // pattern bits ranked at a time (a bitmap of 128 KB)
constexpr int RB_DIGIT = 8;     // sort digit, at most
constexpr int RB_SUB = REFPBWT_SUB;       // sites between the orders the fill pass starts from
constexpr int RB_HIST = 32 * ((1 << RB_DIGIT) + 1);   // digit counts, a row per warp (odd stride: a warp's digits in different banks)

// rows of a block's prefix arrays that hold its scratch
constexpr int RB_ROW_META = 1;   // [0]: ranks of the block, [1]: of the group it starts
constexpr int RB_ROW_KEYS = 2;   // 8 bytes per haplotype (an even row: aligned for any K)
constexpr int RB_ROW_CLS = 4, RB_ROW_GRP = 6;   // ranks of the block, of the group
constexpr int RB_ROW_ORD = 8;    // two orders in flight, where shared memory does not hold them,
constexpr int RB_ROW_DIGIT = 10, RB_ROW_HIST = 11;   // their digits (a byte each) and the CTAs' counts

__device__ __forceinline__ int32_t *rb_row(int32_t *absperm, int K, int block, int row) {
    return absperm + ((size_t)block * RB_SITES + row) * K;
}
__device__ __forceinline__ int rb_width(int n) { return n > 1 ? 32 - __clz(n - 1) : 0; }   // bits of 0 .. n-1

// inclusive scan of one value per thread over the block (1024 threads); ws: 32 ints
__device__ __forceinline__ int rb_scan(int v, int *ws, int *total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) ws[w] = x;
    __syncthreads();
    if (w == 0) {
        int z = ws[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, z, o);
            if (lane >= o) z += y;
        }
        ws[lane] = z;
    }
    __syncthreads();
    if (w) x += ws[w - 1];
    *total = ws[31];
    __syncthreads();
    return x;
}

// Dense ranks.  r holds each haplotype's rank so far (of n values); every turn
// puts the next digit of its key above the rank, marks the values that occur in
// a bitmap and replaces them by their rank among the marked.  group 0: the keys
// of block blockIdx.x; else the ranks of the blocks of group blockIdx.x, first
// block first.  CLS: 16-bit ranks where the haplotypes allow.
template <typename CLS>
__global__ void __launch_bounds__(1024, 1) rp_class_kernel(int32_t *__restrict__ absperm, int K, int nblocks, int group,
                                                           int bits) {
    extern __shared__ uint32_t rc_smem[];
    // the bitmap and the counts before its words, a gap after every 32 words: a
    // thread counts consecutive words, 32 apart from its neighbours'
    const int words = 1 << (bits - 5);
    uint32_t *map = rc_smem;
    uint16_t *off = reinterpret_cast<uint16_t *>(map + words + words / 32 + 1);   // marked before a word, from its thread's first
    int *base = reinterpret_cast<int *>(off + words + 2 * (words / 32 + 1));      // marked before a thread's words
    int *ws = base + 1024;
    const int tid = threadIdx.x;
    const int first = group ? blockIdx.x * group : blockIdx.x;
    const int last = group ? min(first + group, nblocks) : first + 1;
    CLS *r = reinterpret_cast<CLS *>(rb_row(absperm, K, first, group ? RB_ROW_GRP : RB_ROW_CLS));
    int n = 1;
    bool fresh = true;   // no rank yet
    for (int b = first; b < last; b++) {
        const unsigned long long *keys = reinterpret_cast<const unsigned long long *>(rb_row(absperm, K, b, RB_ROW_KEYS));
        const CLS *cls = reinterpret_cast<const CLS *>(rb_row(absperm, K, b, RB_ROW_CLS));
        const int total = group ? rb_width(rb_row(absperm, K, b, RB_ROW_META)[0]) : RB_SITES;
        for (int at = 0; at < total;) {
            const int rb = rb_width(n), db = min(total - at, bits - rb);
            const unsigned long long mask = (1ull << db) - 1ull;
            const int used = max(1, (1 << (rb + db)) >> 5);
            for (int i = tid; i < used + used / 32 + 1; i += 1024) map[i] = 0u;
            __syncthreads();
#pragma unroll 8
            for (int h = tid; h < K; h += 1024) {
                const unsigned d = (unsigned)(((group ? (unsigned long long)cls[h] : keys[h]) >> at) & mask);
                const unsigned code = d << rb | (fresh ? 0u : (unsigned)r[h]);
                atomicOr(&map[(code >> 5) + (code >> 10)], 1u << (code & 31));
            }
            __syncthreads();
            const int per = (used + 1023) / 1024;
            int cnt = 0;
            for (int i = tid * per; i < min(used, (tid + 1) * per); i++) {
                off[i + 2 * (i >> 5)] = (uint16_t)cnt;
                cnt += __popc(map[i + (i >> 5)]);
            }
            int all;
            base[tid] = rb_scan(cnt, ws, &all) - cnt;
            __syncthreads();
#pragma unroll 8
            for (int h = tid; h < K; h += 1024) {
                const unsigned d = (unsigned)(((group ? (unsigned long long)cls[h] : keys[h]) >> at) & mask);
                const unsigned code = d << rb | (fresh ? 0u : (unsigned)r[h]);
                const int w = (int)(code >> 5);
                r[h] = (CLS)(base[w / per] + off[w + 2 * (w >> 5)] + __popc(map[w + (w >> 5)] & ((1u << (code & 31)) - 1u)));
            }
            n = all;
            at += db;
            fresh = false;
            __syncthreads();
        }
    }
    if (fresh)   // one pattern throughout: nothing to rank
        for (int h = tid; h < K; h += 1024) r[h] = (CLS)0;
    if (tid == 0) rb_row(absperm, K, first, RB_ROW_META)[group ? 1 : 0] = n;
}

__host__ __device__ __forceinline__ size_t rc_smem_bytes(int bits) {
    const size_t words = (size_t)1 << (bits - 5);
    return words * 6 + (words / 32 + 1) * 8 + (1024 + 32) * 4;
}

// lanes with this lane's digit, none where !ok.  __match_any_sync takes longer the
// more digits differ: where nearly all do (SPREAD, the ranks of groups) a ballot
// per bit is faster (12 passes over 20,000 haplotypes 0.51 -> 0.31 ms), where few
// do it is not (6 passes by 8 sites' alleles 0.08 -> 0.16 ms).
template <bool SPREAD>
__device__ __forceinline__ unsigned rb_same(unsigned k, bool ok, int db) {
    if (!SPREAD) {
        const unsigned m = __match_any_sync(0xffffffffu, ok ? k : 0x80000000u);
        return ok ? m : 0u;
    }
    unsigned same = __ballot_sync(0xffffffffu, ok);
    for (int j = 0; j < db; j++) {
        const unsigned b = __ballot_sync(0xffffffffu, (k >> j) & 1u);
        same &= (k >> j) & 1u ? b : ~b;
    }
    return ok ? same : 0u;
}

// One stable counting-sort pass of the order by a digit of the ranks: every warp
// counts the digits of its stretch of the order, the counts are scanned
// digit-major, and the warps place their haplotypes in turn.
template <bool SPREAD>
__device__ __forceinline__ void rb_pass(const uint16_t *cur, uint16_t *nxt, const uint16_t *cls, int K, int shift, int db,
                                        int *hist, int *ws) {
    constexpr int U = 2;   // rounds whose lookups run side by side
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int per = ((K + 1023) / 1024) * 32;   // haplotypes of a warp, a multiple of 32
    const int lo = min(K, w * per), hi = min(K, lo + per);
    const unsigned mask = (1u << db) - 1u;
    const int E = 32 << db;
    constexpr int LD = (1 << RB_DIGIT) + 1;
    int *const mine = hist + w * LD;
    for (int i = lane; i <= (int)mask; i += 32) mine[i] = 0;
    __syncthreads();
    for (int i0 = lo; i0 < hi; i0 += 32 * U) {
        unsigned k[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int i = i0 + 32 * u + lane;
            k[u] = i < hi ? (unsigned)cur[i] : 0u;
        }
#pragma unroll
        for (int u = 0; u < U; u++) k[u] = i0 + 32 * u + lane < hi ? ((unsigned)cls[k[u]] >> shift) & mask : mask + 1u;
#pragma unroll
        for (int u = 0; u < U; u++) {
            const unsigned same = rb_same<SPREAD>(k[u], k[u] <= mask, db);
            if (k[u] <= mask && (same & ((1u << lane) - 1u)) == 0u) mine[k[u]] += __popc(same);
            __syncwarp();
        }
    }
    __syncthreads();
    {
        const int n = (E + 1023) / 1024, a = tid * n;
        int v[(32 << RB_DIGIT) / 1024], s = 0;
#pragma unroll
        for (int i = 0; i < (32 << RB_DIGIT) / 1024; i++) {
            v[i] = i < n && a + i < E ? hist[((a + i) & 31) * LD + ((a + i) >> 5)] : 0;
            s += v[i];
        }
        int all;
        int x = rb_scan(s, ws, &all) - s;
#pragma unroll
        for (int i = 0; i < (32 << RB_DIGIT) / 1024; i++)
            if (i < n && a + i < E) { hist[((a + i) & 31) * LD + ((a + i) >> 5)] = x; x += v[i]; }
    }
    __syncthreads();
    for (int i0 = lo; i0 < hi; i0 += 32 * U) {
        unsigned hv[U], k[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int i = i0 + 32 * u + lane;
            hv[u] = i < hi ? (unsigned)cur[i] : 0u;
        }
#pragma unroll
        for (int u = 0; u < U; u++) k[u] = i0 + 32 * u + lane < hi ? ((unsigned)cls[hv[u]] >> shift) & mask : mask + 1u;
#pragma unroll
        for (int u = 0; u < U; u++) {
            const unsigned same = rb_same<SPREAD>(k[u], k[u] <= mask, db);
            const int rank = __popc(same & ((1u << lane) - 1u));
            int at = 0;
            if (k[u] <= mask) {
                at = mine[k[u]];
                nxt[at + rank] = (uint16_t)hv[u];
            }
            __syncwarp();
            if (k[u] <= mask && rank == 0) mine[k[u]] = at + __popc(same);
            __syncwarp();
        }
    }
    __syncthreads();
}

// the order sorted by the ranks of width 'bits' (CTA-wide); cur holds it afterwards
template <bool SPREAD>
__device__ __forceinline__ void rb_sort(uint16_t *&cur, uint16_t *&nxt, const uint16_t *cls, int K, int bits, int *hist,
                                        int *ws) {
    const int passes = (bits + RB_DIGIT - 1) / RB_DIGIT;
    for (int p = 0, at = 0; p < passes; p++) {
        const int db = (bits - at + passes - p - 1) / (passes - p);
        rb_pass<SPREAD>(cur, nxt, cls, K, at, db, hist, ws);
        uint16_t *t = cur; cur = nxt; nxt = t;
        at += db;
    }
}

__host__ __device__ __forceinline__ size_t ro_smem_bytes(int K) { return (size_t)(RB_HIST + 32) * 4 + (size_t)K * 6; }

// TOP: the order before every group, one CTA.  Otherwise: CTA g the orders
// before the blocks of group g after its first.  The two orders and the ranks of
// a step are in shared memory, 16 bits each.
template <bool TOP>
__global__ void __launch_bounds__(1024, 1) rp_order_kernel(int32_t *__restrict__ absperm, int K, int nblocks, int group) {
    extern __shared__ int ro_smem[];
    int *hist = ro_smem, *ws = hist + RB_HIST;
    const int tid = threadIdx.x;
    const int first = TOP ? 0 : blockIdx.x * group;
    const int last = TOP ? nblocks : min(first + group, nblocks);   // blocks first .. last-1 get their order
    const int step = TOP ? group : 1;
    if (!TOP && last - first < 2) return;
    uint16_t *cur = reinterpret_cast<uint16_t *>(ws + 32), *nxt = cur + K, *stage = nxt + K;
    int32_t *start = rb_row(absperm, K, first, 0);
    for (int i = tid; i < K; i += 1024) {
        if (TOP) start[i] = i;
        cur[i] = (uint16_t)(TOP ? i : start[i]);
    }
    __syncthreads();
    for (int b = first; b + step < last; b += step) {
        const uint16_t *cls = reinterpret_cast<const uint16_t *>(rb_row(absperm, K, b, TOP ? RB_ROW_GRP : RB_ROW_CLS));
        for (int i = tid; i < K; i += 1024) stage[i] = cls[i];
        __syncthreads();
        const int bits = rb_width(rb_row(absperm, K, b, RB_ROW_META)[TOP ? 1 : 0]);
        rb_sort<TOP>(cur, nxt, stage, K, bits, hist, ws);
        int32_t *out = rb_row(absperm, K, b + step, 0);
        for (int i = tid; i < K; i += 1024) out[i] = (int32_t)cur[i];
    }
}

// The orders inside a block, every RB_SUB sites, by the alleles themselves (two
// digits): a CTA per block, so that the fill pass has four times as many places to
// start from.
__global__ void __launch_bounds__(1024, 1) rp_sub_kernel(int32_t *__restrict__ absperm, int M, int K) {
    extern __shared__ int ro_smem[];
    int *hist = ro_smem, *ws = hist + RB_HIST;
    const int tid = threadIdx.x, b = blockIdx.x;
    uint16_t *cur = reinterpret_cast<uint16_t *>(ws + 32), *nxt = cur + K, *stage = nxt + K;
    const int32_t *start = rb_row(absperm, K, b, 0);
    const unsigned long long *keys = reinterpret_cast<const unsigned long long *>(rb_row(absperm, K, b, RB_ROW_KEYS));
    for (int i = tid; i < K; i += 1024) cur[i] = (uint16_t)start[i];
    for (int s = 0; s + 1 < RB_SITES / RB_SUB && b * RB_SITES + (s + 1) * RB_SUB < M; s++) {
#pragma unroll 4
        for (int i = tid; i < K; i += 1024) stage[i] = (uint16_t)(keys[i] >> (s * RB_SUB));
        __syncthreads();
        rb_sort<false>(cur, nxt, stage, K, RB_SUB, hist, ws);
        int32_t *out = rb_row(absperm, K, b, (s + 1) * RB_SUB);
        for (int i = tid; i < K; i += 1024) out[i] = (int32_t)cur[i];
    }
}

// Panels whose orders outgrow an SM's shared memory: block after block, each
// sorted by its ranks in passes of RW_DIGIT bits over the whole GPU.  A pass is two
// launches -- every CTA counts the digits of its stretch of the order and
// keeps them, then places its haplotypes after those of the smaller digits
// and of the CTAs before it.  As many passes are launched as the haplotypes'
// number could need; those past a block's ranks return at once.  The first
// pass reads the order before the block, the last writes the order after it.
constexpr int RW_DIGIT = 6, RW_CTAS = 128;

// What pass 'pass' of block b sorts: sub < 0 the block by its ranks, else its
// sites sub * RB_SUB .. by their alleles.  False when there is nothing to do.
__device__ __forceinline__ bool rw_pass(int32_t *absperm, int M, int K, int b, int sub, int pass, int &shift, int &db,
                                        const int32_t *&src, int32_t *&dst) {
    if (sub >= 0 && b * RB_SITES + (sub + 1) * RB_SUB >= M) return false;
    const int bits = sub < 0 ? rb_width(rb_row(absperm, K, b, RB_ROW_META)[0]) : RB_SUB;
    const int passes = max(1, (bits + RW_DIGIT - 1) / RW_DIGIT), from = max(sub, 0) * RB_SUB;
    if (pass >= passes) return false;
    shift = pass * RW_DIGIT;
    db = min(RW_DIGIT, bits - shift);
    src = rb_row(absperm, K, b, pass == 0 ? from : RB_ROW_ORD + ((pass - 1) & 1));
    dst = rb_row(absperm, K, b, pass < passes - 1 ? RB_ROW_ORD + (pass & 1) : sub < 0 ? RB_SITES : from + RB_SUB);
    return true;
}

__global__ void __launch_bounds__(512) rw_count_kernel(int32_t *__restrict__ absperm, int M, int K, int b0, int sub,
                                                       int pass) {
    const int b = b0 + blockIdx.y;
    __shared__ int cnt[1 << RW_DIGIT];
    int shift, db;
    const int32_t *src;
    int32_t *dst;
    if (!rw_pass(absperm, M, K, b, sub, pass, shift, db, src, dst)) return;
    const int32_t *cls = rb_row(absperm, K, b, RB_ROW_CLS);
    const unsigned long long *keys = reinterpret_cast<const unsigned long long *>(rb_row(absperm, K, b, RB_ROW_KEYS));
    const bool first = pass == 0 && b == 0 && sub <= 0;   // the identity order
    uint8_t *digits = reinterpret_cast<uint8_t *>(rb_row(absperm, K, b, RB_ROW_DIGIT));
    int *hist = rb_row(absperm, K, b, RB_ROW_HIST);   // [digit][CTA]
    const int per = (K + RW_CTAS - 1) / RW_CTAS, lo = blockIdx.x * per, hi = min(K, lo + per);
    if (threadIdx.x < (1 << RW_DIGIT)) cnt[threadIdx.x] = 0;
    __syncthreads();
    for (int i = lo + (int)threadIdx.x; i < hi; i += 512) {
        const int h = first ? i : src[i];
        const unsigned d = (sub < 0 ? (unsigned)cls[h] >> shift : (unsigned)(keys[h] >> (sub * RB_SUB + shift))) & ((1u << db) - 1u);
        digits[i] = (uint8_t)d;
        atomicAdd(&cnt[d], 1);
    }
    __syncthreads();
    if (threadIdx.x < (1 << RW_DIGIT)) hist[threadIdx.x * RW_CTAS + blockIdx.x] = cnt[threadIdx.x];
}

__global__ void __launch_bounds__(512) rw_place_kernel(int32_t *__restrict__ absperm, int M, int K, int b0, int sub,
                                                       int pass) {
    const int b = b0 + blockIdx.y;
    __shared__ int base[1 << RW_DIGIT];          // this CTA's next place of each digit
    __shared__ int warpcnt[16][1 << RW_DIGIT];   // of a round of 512: each warp's digits
    int shift, db;
    const int32_t *src;
    int32_t *dst;
    if (!rw_pass(absperm, M, K, b, sub, pass, shift, db, src, dst)) return;
    const uint8_t *digits = reinterpret_cast<const uint8_t *>(rb_row(absperm, K, b, RB_ROW_DIGIT));
    const int *hist = rb_row(absperm, K, b, RB_ROW_HIST);
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const bool first = pass == 0 && b == 0 && sub <= 0;   // the identity order
    const int per = (K + RW_CTAS - 1) / RW_CTAS, lo = blockIdx.x * per, hi = min(K, lo + per);
    // a warp sums a few digits' counts: all of a digit, and of the CTAs before this one
    for (int d = w; d < (1 << RW_DIGIT); d += 16) {
        int all = 0, before = 0;
        for (int c = lane; c < RW_CTAS; c += 32) {
            const int v = hist[d * RW_CTAS + c];
            all += v;
            if (c < (int)blockIdx.x) before += v;
        }
        for (int o = 16; o; o >>= 1) {
            all += __shfl_xor_sync(0xffffffffu, all, o);
            before += __shfl_xor_sync(0xffffffffu, before, o);
        }
        if (lane == 0) { base[d] = before; warpcnt[0][d] = all; }
    }
    __syncthreads();
    if (tid == 0) {
        int run = 0;
        for (int d = 0; d < (1 << RW_DIGIT); d++) {
            const int all = warpcnt[0][d];
            base[d] += run;
            run += all;
        }
    }
    for (int i0 = lo; i0 < hi; i0 += 512) {
        __syncthreads();
        for (int q = tid; q < (16 << RW_DIGIT); q += 512) (&warpcnt[0][0])[q] = 0;
        __syncthreads();
        const int i = i0 + tid;
        const bool ok = i < hi;
        const int h = ok ? (first ? i : src[i]) : 0;
        const unsigned d = ok ? (unsigned)digits[i] : 0u;
        const unsigned same = rb_same<false>(d, ok, db);
        const int rank = __popc(same & ((1u << lane) - 1u));
        if (ok && rank == 0) warpcnt[w][d] = __popc(same);
        __syncthreads();
        if (ok) {
            int at = base[d] + rank;
            for (int q = 0; q < w; q++) at += warpcnt[q][d];
            dst[at] = h;
        }
        __syncthreads();
        if (tid < (1 << RW_DIGIT)) {
            int s = 0;
            for (int q = 0; q < 16; q++) s += warpcnt[q][tid];
            base[tid] += s;
        }
    }
    if (first)   // the order before the first site
        for (int i = lo + tid; i < hi; i += 512) rb_row(absperm, K, 0, 0)[i] = i;
}

// ---------------------------------------------------------------------------
// launcher
// ---------------------------------------------------------------------------


bool refpbwt_by_blocks(int M, int K) {
    // from the second of a block's orders on, and while a digit of at least two bits fits above a
    // rank in the bitmap.  Building a reference on a B200, one-CTA walk and
    // blocks: 100 sites x 2,000 haplotypes 0.29 and 0.20 ms, 200 x 20,000 1.5 and 0.57,
    // 3,000 x 20,000 13 and 1.6, 2,000 x 200,000 (passes over the GPU) 82 and 4.5
    return M > RB_SUB && K >= 64 && K <= (1 << (RB_BITS - 2)) && M / RB_SITES < 65535;
}

cudaError_t launch_refpbwt_blocks(const uint64_t *sitemajor, int M, int K, int wN, int32_t *absperm, cudaStream_t st) {
    int dev = 0, lim = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&lim, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
    if (e != cudaSuccess) return e;
    // the last block's patterns order nothing; its own orders do where it has more than RB_SUB sites
    const int nblocks = (M + RB_SITES - 1) / RB_SITES, ranked = nblocks - 1;
    const bool tail = M - ranked * RB_SITES > RB_SUB;
    const int subs = ranked + (tail ? 1 : 0);
    if ((e = launch_block_keys(sitemajor, tail ? M : ranked * RB_SITES, wN,
                               reinterpret_cast<uint64_t *>(absperm + RB_ROW_KEYS * (size_t)K), K, (size_t)RB_SITES * K / 2,
                               st)) != cudaSuccess)
        return e;
    const size_t rc = rc_smem_bytes(RB_BITS), ro = ro_smem_bytes(K);
    // orders in one SM's shared memory (6 bytes a haplotype beside 33 KB of counts:
    // 33,237 haplotypes on a B200), or passes over the GPU
    if (ro <= (size_t)lim) {
        int group = 2;
        while (group * group < nblocks) group++;
        const int groups = (nblocks + group - 1) / group;   // the last one's patterns order nothing either
        if ((e = ensure_dynamic_smem((const void *)rp_class_kernel<uint16_t>, rc)) != cudaSuccess) return e;
        if (ranked) rp_class_kernel<uint16_t><<<ranked, 1024, rc, st>>>(absperm, K, ranked, 0, RB_BITS);
        if (groups > 1) rp_class_kernel<uint16_t><<<groups - 1, 1024, rc, st>>>(absperm, K, ranked, group, RB_BITS);
        if ((e = ensure_dynamic_smem((const void *)rp_order_kernel<true>, ro)) != cudaSuccess) return e;
        if ((e = ensure_dynamic_smem((const void *)rp_order_kernel<false>, ro)) != cudaSuccess) return e;
        rp_order_kernel<true><<<1, 1024, ro, st>>>(absperm, K, nblocks, group);
        if (ranked) rp_order_kernel<false><<<groups, 1024, ro, st>>>(absperm, K, nblocks, group);
        if ((e = ensure_dynamic_smem((const void *)rp_sub_kernel, ro)) != cudaSuccess) return e;
        rp_sub_kernel<<<subs, 1024, ro, st>>>(absperm, M, K);   // a site count past RB_SUB leaves at least one
        return launched((ranked ? 2 : 0) + (groups > 1 ? 1 : 0) + 2);
    }
    if ((e = ensure_dynamic_smem((const void *)rp_class_kernel<int32_t>, rc)) != cudaSuccess) return e;
    if (ranked) rp_class_kernel<int32_t><<<ranked, 1024, rc, st>>>(absperm, K, ranked, 0, RB_BITS);
    int width = 1;
    while ((1 << width) < K) width++;
    const int rank_passes = (width + RW_DIGIT - 1) / RW_DIGIT, site_passes = (RB_SUB + RW_DIGIT - 1) / RW_DIGIT;
    for (int b = 0; b < ranked; b++)
        for (int p = 0; p < rank_passes; p++) {
            rw_count_kernel<<<RW_CTAS, 512, 0, st>>>(absperm, M, K, b, -1, p);
            rw_place_kernel<<<RW_CTAS, 512, 0, st>>>(absperm, M, K, b, -1, p);
        }
    const dim3 all(RW_CTAS, (unsigned)subs);
    for (int s = 0; s + 1 < RB_SITES / RB_SUB; s++)
        for (int p = 0; p < site_passes; p++) {
            rw_count_kernel<<<all, 512, 0, st>>>(absperm, M, K, 0, s, p);
            rw_place_kernel<<<all, 512, 0, st>>>(absperm, M, K, 0, s, p);
        }
    return launched((ranked ? 1 : 0) + 2 * ranked * rank_passes + 2 * (RB_SITES / RB_SUB - 1) * site_passes);
}

}  // namespace eimp
