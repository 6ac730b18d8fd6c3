// Runs the reference PBWT's checkpoint orders by blocks (generated host copies
// of eimp_b200/csrc/refpbwt_blocks.cu and of the bit transpose of
// imp_kernels.cu) under the warp emulator, whole CTAs one after the other.
//
//   refpbwt_blocks_emu <dir>
//
// <dir> holds params_i.bin (M, K, wN, bits ranked at a time, 16-bit ranks and
// orders in shared memory, blocks per group) and sitemajor.bin (M x wN words).
// Outputs: o_absperm.bin ((M+1) x K int32, the rows of every 16th site) and
// o_trans.bin (K x W(M) words, the transpose).  Exit status 3: a divergent
// warp collective.
#include "refpbwt_blocks_emu.cpp"

#include <string>
#include <thread>
#include <vector>

thread_local dim3 threadIdx, blockIdx, blockDim;
thread_local EmuWarp *emu_warp;
thread_local EmuBarrier *emu_block;
thread_local uint8_t *emu_smem_ptr;
std::atomic<int> emu_divergence{0};

template <class T> static std::vector<T> rd(const std::string &d, const char *name) {
    const std::string p = d + "/" + name;
    FILE *f = fopen(p.c_str(), "rb");
    if (!f) { perror(p.c_str()); exit(1); }
    fseek(f, 0, SEEK_END);
    const long n = ftell(f);
    fseek(f, 0, SEEK_SET);
    std::vector<T> v(n / sizeof(T));
    if (fread(v.data(), 1, n, f) != (size_t)n) exit(2);
    fclose(f);
    return v;
}
template <class T> static void wr(const std::string &d, const char *name, const std::vector<T> &v) {
    const std::string p = d + "/" + name;
    FILE *f = fopen(p.c_str(), "wb");
    if (!f) { perror(p.c_str()); exit(1); }
    fwrite(v.data(), sizeof(T), v.size(), f);
    fclose(f);
}

template <class F> static void run_blocks(int nx, int ny, int nthreads, size_t smem_bytes, F kern) {
    for (int b = 0; b < nx * ny; b++) {
        std::vector<uint64_t> smem((smem_bytes + 7) / 8 + 1, 0x5a5a5a5a5a5a5a5aull);
        std::vector<EmuWarp> warps(nthreads / 32);
        EmuBarrier block;
        block.n = nthreads;
        std::vector<std::thread> threads;
        for (int t = 0; t < nthreads; t++)
            threads.emplace_back([&, t] {
                threadIdx.x = t;
                blockIdx.x = b % nx;
                blockIdx.y = b / nx;
                blockDim.x = nthreads;
                emu_warp = &warps[t / 32];
                emu_block = &block;
                emu_smem_ptr = reinterpret_cast<uint8_t *>(smem.data());
                kern();
            });
        for (auto &x : threads) x.join();
    }
}

template <class CLS> static void orders(const std::vector<uint64_t> &sm, int M, int K, int wN, int bits, bool smem,
                                        int group, std::vector<int32_t> &absperm) {
    using namespace eimp;
    int32_t *ap = absperm.data();
    const int nblocks = (M + RB_SITES - 1) / RB_SITES, ranked = nblocks - 1, groups = (nblocks + group - 1) / group;
    const int ncw = (K + 63) / 64;
    const bool tail = M - ranked * RB_SITES > RB_SUB;
    const int krows = tail ? M : ranked * 64, subs = ranked + tail;
    run_blocks((krows + TR_ROWS - 1) / TR_ROWS, (ncw + TR_WORDS - 1) / TR_WORDS, TR_ROWS, TR_SMEM, [&] {
        transpose_kernel<true>(sm.data(), (size_t)krows, wN, reinterpret_cast<uint64_t *>(ap + RB_ROW_KEYS * (size_t)K), K,
                               (krows + 63) / 64, (size_t)RB_SITES * K / 2);
    });
    const size_t cs = rc_smem_bytes(bits);
    if (ranked) run_blocks(ranked, 1, 1024, cs, [&] { rp_class_kernel<CLS>(ap, K, ranked, 0, bits); });
    if (!smem) {
        int width = 1;
        while ((1 << width) < K) width++;
        for (int b = 0; b < ranked; b++)
            for (int p = 0; p < (width + RW_DIGIT - 1) / RW_DIGIT; p++) {
                run_blocks(RW_CTAS, 1, 512, 8, [&] { rw_count_kernel(ap, M, K, b, -1, p); });
                run_blocks(RW_CTAS, 1, 512, 8, [&] { rw_place_kernel(ap, M, K, b, -1, p); });
            }
        for (int s = 0; s + 1 < RB_SITES / RB_SUB; s++)
            for (int p = 0; p < (RB_SUB + RW_DIGIT - 1) / RW_DIGIT; p++) {
                run_blocks(RW_CTAS, subs, 512, 8, [&] { rw_count_kernel(ap, M, K, 0, s, p); });
                run_blocks(RW_CTAS, subs, 512, 8, [&] { rw_place_kernel(ap, M, K, 0, s, p); });
            }
        return;
    }
    if (groups > 1) run_blocks(groups - 1, 1, 1024, cs, [&] { rp_class_kernel<CLS>(ap, K, ranked, group, bits); });
    const size_t os = ro_smem_bytes(K);
    run_blocks(1, 1, 1024, os, [&] { rp_order_kernel<true>(ap, K, nblocks, group); });
    if (ranked) run_blocks(groups, 1, 1024, os, [&] { rp_order_kernel<false>(ap, K, nblocks, group); });
    run_blocks(subs, 1, 1024, os, [&] { rp_sub_kernel(ap, M, K); });
}

int main(int argc, char **argv) {
    if (argc < 2) { fprintf(stderr, "usage: %s <dir>\n", argv[0]); return 1; }
    const std::string d = argv[1];
    const auto pi = rd<int32_t>(d, "params_i.bin");
    const int M = pi[0], K = pi[1], wN = pi[2], bits = pi[3], smem = pi[4], group = pi[5];
    const auto sm = rd<uint64_t>(d, "sitemajor.bin");
    std::vector<int32_t> absperm((size_t)(M + 1) * K, -1);
    if (smem) orders<uint16_t>(sm, M, K, wN, bits, true, group, absperm);
    else orders<int32_t>(sm, M, K, wN, bits, false, group, absperm);
    wr(d, "o_absperm.bin", absperm);
    const int wM = (int)eimp_W(M);
    std::vector<uint64_t> tr((size_t)K * wM, 0xdeadbeefdeadbeefull);
    run_blocks((wM * 64 + eimp::TR_ROWS - 1) / eimp::TR_ROWS, ((K + 63) / 64 + eimp::TR_WORDS - 1) / eimp::TR_WORDS, eimp::TR_ROWS,
               eimp::TR_SMEM, [&] { eimp::transpose_kernel<false>(sm.data(), M, wN, tr.data(), K, wM, wM); });
    wr(d, "o_trans.bin", tr);
    if (emu_divergence.load()) { fprintf(stderr, "divergent warp collectives: %d\n", emu_divergence.load()); return 3; }
    return 0;
}
