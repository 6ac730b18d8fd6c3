// Runs smm_list_kernel (generated host copy of eimp_b200/csrc/smm_list.cu)
// under the warp emulator, whole CTAs one after the other.
//
//   smm_list_emu <dir> <wide> <warps> <group> <pool slots> [chunks]
//
// <dir> holds params_i.bin (nhaps, M, K, cap, nrows, use_hapmap), compr.bin,
// phased.bin, gt.bin and hapmap.bin as smm_main.cpp takes them; wide: 64-bit
// intervals; warps: haplotypes per CTA; group: rows per ring stage (0: read
// in place); chunks: parts of a haplotype's sites, joined by
// smm_list_join_kernel when there are several.  Outputs: o_matches.bin, o_nmatch.bin, o_status.bin (status,
// pool slots taken).  Exit status 3: a divergent warp collective.
#include "smm_list_emu.cpp"

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

template <bool WIDE> static int go(const std::string &d, int warps, int group, int slots, int chunks) {
    using namespace eimp;
    const auto pi = rd<int32_t>(d, "params_i.bin");
    const int nhaps = pi[0], M = pi[1], K = pi[2], cap = pi[3], nrows = pi[4];
    const std::vector<int32_t> hapmap = pi[5] ? rd<int32_t>(d, "hapmap.bin") : std::vector<int32_t>();
    const auto rows = rd<uint32_t>(d, "compr.bin");
    // aligned like device memory and readable up to the next 16-byte boundary past the end, no further
    const size_t bytes = (rows.size() * 4 + 15) / 16 * 16;
    uint32_t *compr = (uint32_t *)aligned_alloc(16, bytes);
    memset(compr, 0x5A, bytes);
    memcpy(compr, rows.data(), rows.size() * 4);
    const auto phased = rd<uint64_t>(d, "phased.bin");
    const auto gt = rd<uint8_t>(d, "gt.bin");
    std::vector<int4> matches((size_t)nrows * cap, int4{-7, -7, -7, -7});
    std::vector<int32_t> nmatch(nrows, -7);
    uint32_t status = 0;
    int gnext = 0;
    typedef SlList<WIDE, SL_POOL> Pool;
    std::vector<uint64_t> gpool(slots * sizeof(Pool) / 8, 0x5a5a5a5a5a5a5a5aull);
    const size_t rowbytes = (size_t)((K + 31) / 32) * 8, stage = group ? (group * rowbytes + 30) & ~(size_t)15 : 0;
    const size_t smb = SL_HEAD + SL_STAGES * stage + (size_t)warps * sizeof(SlList<WIDE, SL_CAP>);
    const int nthreads = 32 * (warps + (group ? 1 : 0));
    for (int b = 0; b < (nhaps + warps - 1) / warps; b++) for (int chunk = 0; chunk < chunks; chunk++) {
        uint8_t *smem = (uint8_t *)aligned_alloc(16, (smb + 15) / 16 * 16);
        memset(smem, 0x5A, smb);
        std::vector<EmuWarp> ws(nthreads / 32);
        EmuBarrier block;
        block.n = nthreads;
        std::vector<std::thread> lanes;
        for (int t = 0; t < nthreads; t++)
            lanes.emplace_back([&, t] {
                threadIdx.x = t;
                blockIdx.x = b;
                blockIdx.y = chunk;
                blockDim.x = nthreads;
                emu_warp = &ws[t / 32];
                emu_block = &block;
                emu_smem_ptr = smem;
                smm_list_kernel<WIDE>(compr, M, K, phased.data(), (int)eimp_W(M), gt.data(), nhaps,
                                      hapmap.empty() ? nullptr : hapmap.data(), matches.data(), cap, nmatch.data(),
                                      &status, warps, group, (unsigned)stage, slots ? (Pool *)gpool.data() : nullptr,
                                      slots, &gnext, chunks);
            });
        for (auto &x : lanes) x.join();
        free(smem);
    }
    for (int b = 0; chunks > 1 && b < nhaps; b++) {
        EmuWarp w;
        std::vector<std::thread> lanes;
        for (int t = 0; t < 32; t++)
            lanes.emplace_back([&, t] {
                threadIdx.x = t;
                blockIdx.x = b;
                blockDim.x = 32;
                emu_warp = &w;
                smm_list_join_kernel(M, hapmap.empty() ? nullptr : hapmap.data(), matches.data(), cap, nmatch.data(),
                                     &status, chunks);
            });
        for (auto &x : lanes) x.join();
    }
    free(compr);
    wr(d, "o_matches.bin", matches);
    wr(d, "o_nmatch.bin", nmatch);
    wr(d, "o_status.bin", std::vector<int32_t>{(int)status, gnext});
    if (emu_divergence.load()) { fprintf(stderr, "divergent warp collectives: %d\n", emu_divergence.load()); return 3; }
    return 0;
}

int main(int argc, char **argv) {
    if (argc < 6) { fprintf(stderr, "usage: %s <dir> <wide> <warps> <group> <slots> [chunks]\n", argv[0]); return 1; }
    const int warps = atoi(argv[3]), group = atoi(argv[4]), slots = atoi(argv[5]);
    const int chunks = argc > 6 ? atoi(argv[6]) : 1;
    return atoi(argv[2]) ? go<true>(argv[1], warps, group, slots, chunks) : go<false>(argv[1], warps, group, slots, chunks);
}
