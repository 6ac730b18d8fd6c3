"""The match search without mismatches (eimp_b200/csrc/smm_list.cu) on the
CPU under the warp emulator, with the address and undefined-behaviour
sanitizers, against the oracle restatement of TargetImp::calcSMMatches: rows
through the ring (groups that end off the row count, row sizes off 16 bytes)
and in place, narrow and wide intervals, CTAs of one and several haplotypes, a
row map, lists that move to a global pool or outgrow the list, a match buffer
that is too small, and targets with more than half their sites missing."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT, golden_path
from eimp_b200.bits import W, pack_rows

CSRC = os.path.join(ROOT, "eimp_b200", "csrc")
EMU = os.path.join(ROOT, "tests", "warp_emu")


@pytest.fixture(scope="module")
def emu_exe(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    d = tmp_path_factory.mktemp("smm_list_emu")
    for f in ("common.cuh", "kernels.h"):
        shutil.copy(os.path.join(CSRC, f), d / f)
    src = open(os.path.join(CSRC, "smm_list.cu")).read()
    j = src.index("// launcher\n")
    src = src[:src.rindex("// ----", 0, j)] + "}\n"
    decl = "extern __shared__ __align__(16) uint8_t smem_raw[];"
    assert decl in src
    (d / "smm_list_emu.cpp").write_text('#include "emu.h"\n' + src.replace(decl, "uint8_t *smem_raw = emu_smem_ptr;"))
    exe = d / "smm_list_emu"
    r = subprocess.run(["g++", "-std=c++20", "-O1", "-g", "-fsanitize=address,undefined",
                        "-fno-sanitize-recover=undefined", "-I", EMU, "-I", str(d),
                        os.path.join(EMU, "smm_list_main.cpp"), "-o", str(exe), "-lpthread"],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    return str(exe)


def run(exe, d, compr, phased, gt, K, wide, warps, group, slots=0, cap=None, hapmap=None, chunks=1):
    nrows, M = phased.shape[0], gt.shape[1]
    cap = cap or M + 64
    nh = nrows if hapmap is None else len(hapmap)
    os.makedirs(d, exist_ok=True)
    for name, a in [("params_i", np.array([nh, M, K, cap, nrows, hapmap is not None], np.int32)),
                    ("compr", compr.astype(np.uint32)), ("phased", phased.astype(np.uint64)),
                    ("gt", gt.astype(np.uint8)),
                    ("hapmap", np.asarray([0] if hapmap is None else hapmap, np.int32))]:
        np.ascontiguousarray(a).tofile(os.path.join(d, name + ".bin"))
    r = subprocess.run([exe, str(d), str(int(wide)), str(warps), str(group), str(slots), str(chunks)], capture_output=True,
                       text=True, timeout=900)
    assert r.returncode == 0, f"rc {r.returncode}: {r.stderr[-4000:]}"
    m = np.fromfile(os.path.join(d, "o_matches.bin"), np.int32).reshape(nrows, cap, 4).astype(np.int64)
    n = np.fromfile(os.path.join(d, "o_nmatch.bin"), np.int32)
    status, moved = (int(x) for x in np.fromfile(os.path.join(d, "o_status.bin"), np.int32))
    return m, n, status, moved


def panel(rng, M, K, F, err=0.01):
    """Site-major rows of K mosaics of F founders, and four targets of the
    same kind as haplotype rows."""
    f = rng.random((F, M)) < rng.choice([0.02, 0.3, 0.5], M)
    n = K + 8
    src = np.zeros((n, M), np.int64)
    src[:, 0] = rng.integers(0, F, n)
    sw = rng.random((n, M)) < 0.03
    for m in range(1, M):
        src[:, m] = np.where(sw[:, m], rng.integers(0, F, n), src[:, m - 1])
    h = (f[src, np.arange(M)] ^ (rng.random((n, M)) < err)).astype(np.uint8)
    return pack_rows(np.ascontiguousarray(h[:K].T), W(K)), h[K:]


@pytest.mark.parametrize("K,M,wide,warps,group", [(64, 1, 0, 1, 1), (33, 150, 0, 3, 4), (700, 203, 0, 8, 3),
                                                  (700, 203, 1, 2, 0), (1000, 97, 0, 4, 16), (320, 64, 1, 4, 0)])
def test_against_oracle(emu_exe, tmp_path, K, M, wide, warps, group):
    from oracle import restate as R
    rng = np.random.default_rng(K * 31 + M)
    sm, th = panel(rng, M, K, 12)
    gt = np.where(rng.random((4, M)) < 0.06, 3, th[0::2] + th[1::2]).astype(np.uint8)
    gt[3, rng.permutation(M)[:M // 2 + 1]] = 3
    ph = pack_rows(th, W(M))
    compr, c0, _ = R.pbwt(sm, K)
    m, n, status, moved = run(emu_exe, tmp_path / "k", compr, ph, gt, K, wide, warps, group)
    assert status == 0 and moved == 0
    for h in range(8):
        om = R.smmatches(compr, c0, M, K, ph[h], np.flatnonzero(gt[h // 2] == 3).astype(np.int64))
        assert n[h] == len(om)
        np.testing.assert_array_equal(m[h, :n[h]], om)


@pytest.mark.parametrize("wide,group", [(0, 2), (1, 0)])
def test_large_lists(emu_exe, tmp_path, wide, group):
    """Runs of missing sites on an unstructured panel: the lists outgrow
    shared memory and move to a pool; without a pool left the haplotype gets
    the retry mark, and the others are not affected."""
    from oracle import restate as R
    rng = np.random.default_rng(5)
    K, M = 2200, 48
    sm = pack_rows((rng.random((M, K)) < 0.5).astype(np.uint8), W(K))
    gt = rng.integers(0, 2, (2, M)).astype(np.uint8)
    gt[0, 8:17] = 3
    gt[0, 30:40] = 3
    ph = pack_rows((rng.random((4, M)) < 0.5).astype(np.uint8), W(M))
    compr, c0, _ = R.pbwt(sm, K)
    for slots, marked in ((2, 0), (1, 1), (0, 2)):
        m, n, status, moved = run(emu_exe, tmp_path / f"k{slots}", compr, ph, gt, K, wide, 4, group, slots)
        assert status == 0 and moved == (2 if slots else 0) and (n == -2).sum() == marked
        for h in range(4):
            if n[h] == -2:
                continue
            om = R.smmatches(compr, c0, M, K, ph[h], np.flatnonzero(gt[h // 2] == 3).astype(np.int64))
            assert n[h] == len(om)
            np.testing.assert_array_equal(m[h, :n[h]], om)


def test_move_at_every_offset(emu_exe, tmp_path):
    """A list moves to its pool at any site, the first of 32 among them (the
    genotypes and alleles are read 32 sites at a time)."""
    from oracle import restate as R
    rng = np.random.default_rng(6)
    K, M = 1200, 72
    sm = pack_rows((rng.random((M, K)) < 0.5).astype(np.uint8), W(K))
    gt = rng.integers(0, 2, (6, M)).astype(np.uint8)
    for t in range(6):
        gt[t, 21 + t:30 + t] = 3
    ph = pack_rows((rng.random((12, M)) < 0.5).astype(np.uint8), W(M))
    compr, c0, _ = R.pbwt(sm, K)
    m, n, status, moved = run(emu_exe, tmp_path / "k", compr, ph, gt, K, 0, 4, 5, 12)
    assert status == 0 and moved == 12
    for h in range(12):
        om = R.smmatches(compr, c0, M, K, ph[h], np.flatnonzero(gt[h // 2] == 3).astype(np.int64))
        assert n[h] == len(om)
        np.testing.assert_array_equal(m[h, :n[h]], om)


def test_match_buffer_too_small(emu_exe, tmp_path):
    from oracle import restate as R
    rng = np.random.default_rng(9)
    K, M = 200, 120
    sm, th = panel(rng, M, K, 6)
    gt = (th[0::2] + th[1::2]).astype(np.uint8)
    compr, _, _ = R.pbwt(sm, K)
    _, n, status, _ = run(emu_exe, tmp_path / "k", compr, pack_rows(th, W(M)), gt, K, 0, 8, 4, cap=2)
    assert status == 1 and (n == -1).all()


@pytest.mark.parametrize("K,M,wide,warps,group,chunks,err", [(64, 7, 0, 1, 1, 2, 0.0), (300, 150, 0, 3, 4, 3, 0.01),
                                                             (700, 203, 0, 8, 3, 13, 0.003), (700, 203, 1, 2, 0, 32, 0.01),
                                                             (500, 320, 0, 5, 16, 10, 0.0), (500, 96, 1, 4, 0, 3, 0.0)])
def test_chunks_against_oracle(emu_exe, tmp_path, K, M, wide, warps, group, chunks, err):
    """A haplotype's sites in parts: matches across one and several of their
    boundaries, one over all sites (a copy of a panel haplotype), parts
    without a match of their own, sites missing at and around a boundary."""
    from oracle import restate as R
    rng = np.random.default_rng(K * 31 + M + chunks)
    sm, th = panel(rng, M, K, 12, err)
    th[0] = (sm.reshape(M, -1)[:, 5 // 64] >> np.uint64(5)) & np.uint64(1)
    gt = np.where(rng.random((4, M)) < 0.06, 3, th[0::2] + th[1::2]).astype(np.uint8)
    gt[1, M // chunks - 1:M // chunks + 2] = 3
    gt[3, rng.permutation(M)[:M // 2 + 1]] = 3
    ph = pack_rows(th, W(M))
    compr, c0, _ = R.pbwt(sm, K)
    hapmap = [0, 3, 2, 4, 7]
    m, n, status, _ = run(emu_exe, tmp_path / "k", compr, ph, gt, K, wide, warps, group, hapmap=hapmap, chunks=chunks,
                          cap=chunks * (M + 2))
    assert status == 0
    for h in hapmap:
        om = R.smmatches(compr, c0, M, K, ph[h], np.flatnonzero(gt[h // 2] == 3).astype(np.int64))
        assert n[h] == len(om)
        np.testing.assert_array_equal(m[h, :n[h]], om)
    assert (n[[1, 5, 6]] == -7).all()


@pytest.mark.parametrize("wide,group", [(0, 2), (1, 0)])
def test_chunks_that_cannot_be_joined(emu_exe, tmp_path, wide, group):
    """Lists that outgrow a chunk's, or that together could outgrow the most a
    list may hold, and a part of the buffer that is too small: the haplotype
    gets the retry mark."""
    from oracle import restate as R
    rng = np.random.default_rng(15)
    K, M = 2200, 96
    sm = pack_rows((rng.random((M, K)) < 0.5).astype(np.uint8), W(K))
    gt = rng.integers(0, 2, (2, M)).astype(np.uint8)
    gt[0, 8:17] = 3
    gt[0, 70:80] = 3
    ph = pack_rows((rng.random((4, M)) < 0.5).astype(np.uint8), W(M))
    compr, c0, _ = R.pbwt(sm, K)
    want = [R.smmatches(compr, c0, M, K, ph[h], np.flatnonzero(gt[h // 2] == 3).astype(np.int64)) for h in range(4)]
    for slots, again in ((8, []), (0, [0, 1])):
        m, n, status, _ = run(emu_exe, tmp_path / f"k{slots}", compr, ph, gt, K, wide, 4, group, slots, chunks=2)
        assert status == 0 and list(np.flatnonzero(n == -2)) == again
        for h in set(range(4)) - set(again):
            assert n[h] == len(want[h])
            np.testing.assert_array_equal(m[h, :n[h]], want[h])
    _, n, status, _ = run(emu_exe, tmp_path / "small", compr, ph, gt, K, wide, 4, group, 8, cap=6, chunks=3)
    assert status == 0 and (n[2:] == -2).all()
    gt[0, 8:21] = 3    # more than 4,096 entries in one piece
    gt[0, 70:83] = 3
    _, n, status, _ = run(emu_exe, tmp_path / "large", compr, ph, gt, K, wide, 4, group, 8, chunks=2)
    one = run(emu_exe, tmp_path / "one", compr, ph, gt, K, wide, 4, group, 8)
    assert ((one[1] == -2) <= (n == -2)).all() and status == one[2] == 0


def test_haploid_golden(emu_exe, tmp_path):
    """The reference's own matches of the haploid golden case (a row map)."""
    g = np.load(golden_path("golden_haploid.npz"))
    gt = np.ascontiguousarray(g["gt"], np.uint8)
    nt, M = gt.shape
    K = int(g["imp_K"])
    hapmap = [h for t in range(nt) for h in ([2 * t] if g["tgt_haploid"][t] else [2 * t, 2 * t + 1])]
    m, n, status, _ = run(emu_exe, tmp_path / "k", g["imp_compr"], g["imp_phased"], gt, K, 0, 5, 7, hapmap=hapmap)
    assert status == 0
    off = np.concatenate([[0], np.cumsum(g["imp_nmatches"])])
    for j, h in enumerate(hapmap):
        np.testing.assert_array_equal(m[h, :n[h]], g["imp_matches"][off[j]:off[j + 1]])
