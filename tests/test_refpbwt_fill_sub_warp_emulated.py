"""The reference PBWT's fill pass from the orders before every 16th site
(refpbwt_fill_sub_kernel in eimp_b200/csrc/imp_kernels.cu), one and four words
of the order at a time, on the CPU under the warp emulator with the
sanitizers: compressed rows, prefix arrays and zero counts against the oracle,
with site counts on and off a multiple of 16 and orders of one and several
rounds of a warp's words."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from eimp_b200.bits import W
from test_refpbwt_warp_emulated import CSRC, EMU


@pytest.fixture(scope="module")
def emu_exe(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    d = tmp_path_factory.mktemp("refpbwt_fill_emu")
    for f in ("common.cuh", "kernels.h"):
        shutil.copy(os.path.join(CSRC, f), d / f)
    src = open(os.path.join(CSRC, "imp_kernels.cu")).read()
    i = src.rindex("// ----", 0, src.index("// block-wide exclusive scan"))
    j = src.rindex("// ----", 0, src.index("// bit-matrix transpose"))
    body = src[i:j]
    for a, b, n in [("extern __shared__ uint64_t rp_smem[];",
                     "uint64_t *rp_smem = reinterpret_cast<uint64_t *>(emu_smem_ptr);", 1),
                    ("extern __shared__ uint8_t smem[];", "uint8_t *smem = emu_smem_ptr;", 2)]:
        assert body.count(a) == n
        body = body.replace(a, b)
    (d / "refpbwt_emu.cpp").write_text('#include "emu.h"\n#include "common.cuh"\n#include "kernels.h"\n'
                                       "namespace eimp {\n" + body + "}  // namespace eimp\n")
    main = open(os.path.join(EMU, "refpbwt_main.cpp")).read()
    # the orders before every 16th site in place of the checkpoint pass
    i, j = main.index("    std::vector<int32_t> scratch("), main.index("    const size_t fill_smem")
    main = main[:i] + """    const auto orders = rd<int32_t>(d, "orders.bin");
    for (int m = 0; m < M; m += eimp::RP_SUB)
        std::copy(orders.begin() + (size_t)(m / eimp::RP_SUB) * K, orders.begin() + (size_t)(m / eimp::RP_SUB + 1) * K,
                  absperm.begin() + (size_t)m * K);
    (void)in_smem;
""" + main[j:]
    for a, b in [("eimp::RP_CK - 1) / eimp::RP_CK", "eimp::RP_SUB - 1) / eimp::RP_SUB"),
                 ("eimp::refpbwt_fill_kernel(sm.data(), M, K, wN, compr.data(), absperm.data(), count0.data());",
                  "(stage == 4 ? eimp::refpbwt_fill_sub_kernel<4> : eimp::refpbwt_fill_sub_kernel<1>)"
                  "(sm.data(), M, K, wN, compr.data(), absperm.data(), count0.data());")]:
        assert main.count(a) == 1
        main = main.replace(a, b)
    (d / "main.cpp").write_text("#include <algorithm>\n" + main)
    exe = d / "refpbwt_emu"
    r = subprocess.run(["g++", "-std=c++20", "-O1", "-g", "-fsanitize=address,undefined",
                        "-fno-sanitize-recover=undefined", "-I", EMU, "-I", str(d), str(d / "main.cpp"), "-o",
                        str(exe), "-lpthread"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    return str(exe)


@pytest.mark.parametrize("M,K", [(17, 64), (32, 1024), (37, 1100), (16, 4097), (21, 5000)])
@pytest.mark.parametrize("words", [1, 4])
def test_fill_from_block_orders(emu_exe, tmp_path, M, K, words):
    from oracle import restate as R
    rng = np.random.default_rng(M * 7919 + K)
    wN = W(K)
    dens = rng.choice([0.0, 0.01, 0.2, 0.5, 1.0], size=M, p=[0.05, 0.3, 0.3, 0.3, 0.05])
    bits = (rng.random((M, wN * 64)) < dens[:, None]).astype(np.uint8)
    bits[:, K:] = rng.integers(0, 2, (M, wN * 64 - K))   # padding past K is never read
    sm = np.packbits(bits, axis=1, bitorder="little").view(np.uint64).reshape(M, wN)
    rc, rc0, rap = R.pbwt(np.ascontiguousarray(sm), K, absperm=True)
    np.array([M, K, wN, 0, words], np.int32).tofile(tmp_path / "params_i.bin")
    sm.tofile(tmp_path / "sitemajor.bin")
    np.ascontiguousarray(rap[0:M:16], np.int32).tofile(tmp_path / "orders.bin")
    r = subprocess.run([emu_exe, str(tmp_path)], capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, f"rc {r.returncode}: {r.stderr[-4000:]}"
    compr = np.fromfile(tmp_path / "o_compr.bin", np.uint32).reshape(M, 2 * ((K + 31) // 32))
    ap = np.fromfile(tmp_path / "o_absperm.bin", np.int32).reshape(M + 1, K)
    c0 = np.fromfile(tmp_path / "o_count0.bin", np.int32)
    np.testing.assert_array_equal(ap, rap)
    np.testing.assert_array_equal(compr, rc)
    np.testing.assert_array_equal(c0, rc0)
