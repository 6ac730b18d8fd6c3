"""The reference PBWT's checkpoint orders by blocks of sites
(eimp_b200/csrc/refpbwt_blocks.cu) and the bit transpose (imp_kernels.cu) on the
CPU under the warp emulator, with the sanitizers: the order before every 16th
site against the oracle restatement of PBWT::buildComprPBWT, with 16-bit ranks
and orders in shared memory and with 32-bit ones and passes over many CTAs, ranks taken a few
pattern bits at a time, blocks in which all haplotypes agree (no bits to rank,
the first of a group among them), and site counts on and off a block's end."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT
from eimp_b200.bits import W, transpose_bits

CSRC = os.path.join(ROOT, "eimp_b200", "csrc")
EMU = os.path.join(ROOT, "tests", "warp_emu")


@pytest.fixture(scope="module")
def emu_exe(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    d = tmp_path_factory.mktemp("refpbwt_blocks_emu")
    for f in ("common.cuh", "kernels.h"):
        shutil.copy(os.path.join(CSRC, f), d / f)
    imp = open(os.path.join(CSRC, "imp_kernels.cu")).read()
    i, j = imp.index("constexpr int TR_ROWS"), imp.index("// set-maximal matches\n//\n")
    src = open(os.path.join(CSRC, "refpbwt_blocks.cu")).read()
    src = src[:src.rindex("// ----", 0, src.index("// launcher\n"))]
    assert src.count("RW_CTAS = 128;") == 1
    src = src.replace("RW_CTAS = 128;", "RW_CTAS = 5;")   # several rounds of 512 haplotypes to a CTA
    for k, t, n in (("rc_smem", "uint32_t", 1), ("ro_smem", "int", 2)):
        decl = f"extern __shared__ {t} {k}[];"
        assert src.count(decl) == n
        src = src.replace(decl, f"{t} *{k} = reinterpret_cast<{t} *>(emu_smem_ptr);")
    imp = imp[i:imp.rindex("// ----", 0, j)]
    decl = "extern __shared__ uint32_t tr_smem[];"
    assert imp.count(decl) == 1
    imp = imp.replace(decl, "uint32_t *tr_smem = reinterpret_cast<uint32_t *>(emu_smem_ptr);")
    (d / "refpbwt_blocks_emu.cpp").write_text('#include "emu.h"\n' + src + imp + "}\n")
    exe = d / "refpbwt_blocks_emu"
    r = subprocess.run(["g++", "-std=c++20", "-O1", "-g", "-fsanitize=address,undefined",
                        "-fno-sanitize-recover=undefined", "-I", EMU, "-I", str(d),
                        os.path.join(EMU, "refpbwt_blocks_main.cpp"), "-o", str(exe), "-lpthread"],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    return str(exe)


@pytest.mark.parametrize("M,K,smem,bits,group", [(17, 90, 1, 14, 2), (40, 2700, 0, 14, 2), (81, 66, 1, 9, 2), (256, 300, 1, 14, 2), (300, 1100, 1, 13, 3), (250, 5000, 0, 15, 2),
                                                 (193, 2700, 0, 17, 3), (321, 1500, 1, 20, 4)])
def test_orders(emu_exe, tmp_path, M, K, smem, bits, group):
    from oracle import restate as R
    rng = np.random.default_rng(M * 7919 + K)
    wN = W(K)
    dens = rng.choice([0.0, 0.01, 0.2, 0.5, 1.0], size=M, p=[0.05, 0.3, 0.3, 0.3, 0.05])
    founders = rng.random((M, 40)) < dens[:, None]
    h = founders[:, rng.integers(0, 40, K)] ^ (rng.random((M, K)) < 0.002)
    if M > 200:
        h[:64] = rng.random((64, 1)) < 0.5          # every haplotype the same: nothing to rank
    if M > 320:
        h[192:256] = h[192:256, :1]
    b = np.zeros((M, wN * 64), np.uint8)
    b[:, :K] = h
    b[:, K:] = rng.integers(0, 2, (M, wN * 64 - K))   # padding past K is never read
    sm = np.packbits(b, axis=1, bitorder="little").view(np.uint64).reshape(M, wN)
    np.array([M, K, wN, bits, smem, group], np.int32).tofile(tmp_path / "params_i.bin")
    sm.tofile(tmp_path / "sitemajor.bin")
    r = subprocess.run([emu_exe, str(tmp_path)], capture_output=True, text=True, timeout=900)
    assert r.returncode == 0, f"rc {r.returncode}: {r.stderr[-4000:]}"
    got = np.fromfile(tmp_path / "o_absperm.bin", np.int32).reshape(M + 1, K)
    _, _, want = R.pbwt(sm, K, absperm=True)
    for m in range(0, M, 16):
        np.testing.assert_array_equal(got[m], want[m])
    tr = np.fromfile(tmp_path / "o_trans.bin", np.uint64).reshape(K, W(M))
    np.testing.assert_array_equal(tr, transpose_bits(sm, M, K))
