"""The beam kernel's several warps under the warp emulator built with the thread
sanitizer: nothing may be written by one lane and read or written by another
without a warp or block barrier between.  With every haplotype path in the
arena, whose interval pool is the constraint heaps' storage after the
pre-phasing pass, and a fast look-ahead of 0 (delta_fast), so that the last
call of that pass has advanced the beam and its splitting paths are still
being copied when the heaps are to be filled."""
import os
import re
import shutil
import subprocess

import numpy as np
import pytest

from conftest import golden_path
from test_beam_warp_emulated import CSRC, EMU, golden_inputs, write_inputs

WARPS = 4


@pytest.fixture(scope="module")
def emu_exe(tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    d = tmp_path_factory.mktemp("beam_races_emu")
    for f in ("common.cuh", "kernels.h"):
        shutil.copy(os.path.join(CSRC, f), d / f)
    src = open(os.path.join(CSRC, "beam.cu")).read()
    i, j = src.index("static size_t beam_smem("), src.rindex("}  // namespace eimp")
    decl = "extern __shared__ __align__(16) uint8_t smem_raw[];"
    assert src.count(decl) == 1
    src = (src[:i] + src[j:]).replace(decl, "uint8_t *smem_raw = emu_smem_ptr;")
    (d / "beam_emu.cpp").write_text('#include "emu.h"\n' + src)
    main = open(os.path.join(EMU, "beam_main.cpp")).read()
    for old, new, n in [
            ("eimp::beam_canon_bytes(al.NH);", f"eimp::beam_canon_bytes(al.NH) + eimp::beam_term_bytes({WARPS});", 1),
            ("EmuWarp warp;", f"std::vector<EmuWarp> warps({WARPS}); EmuBarrier block; block.n = {32 * WARPS};", 2),
            ("l < 32;", f"l < {32 * WARPS};", 2), ("blockDim.x = 32;", f"blockDim.x = {32 * WARPS};", 2),
            ("emu_warp = &warp;", "emu_warp = &warps[l / 32]; emu_block = &block;", 2)]:
        assert main.count(old) == n
        main = main.replace(old, new)
    (d / "main.cpp").write_text(main)
    exe = d / "beam_emu"
    r = subprocess.run(["g++", "-std=c++20", "-O1", "-g", "-ffp-contract=off", "-fno-fast-math", "-fsanitize=thread",
                        "-I", EMU, "-I", str(d), str(d / "main.cpp"), "-o", str(exe), "-lpthread"],
                       capture_output=True, text=True)
    if r.returncode and "tsan" in r.stderr:
        pytest.skip("no thread sanitizer runtime")
    assert r.returncode == 0, r.stderr[-4000:]
    return str(exe)


def reports(exe, d, P, prephase, cuts, H=8):
    """The sanitizer's reports, as lists of the functions on their stacks, for
    the panel's first target cut after each of the given numbers of split
    sites."""
    from oracle import restate as R
    if not R.available():
        pytest.skip("oracle library not built")
    g = np.load(golden_path("golden_tiny.npz"))
    hm, sm, K = g["hapmajor_typed"], g["sitemajor_typed"], 200
    gt = np.ascontiguousarray(g["gt"][0], np.uint8)
    bh, _ = R.besthaps(gt, hm, K)
    mo = R.monos(hm, len(gt), bh)
    sp, ca, cd = R.calllocs(gt, mo, g["cm_typed"])
    crefs = [R.cref(gt, sm, int(g["nhaps"]), bh, sp[:s])[0] for s in cuts]
    n = len(cuts)
    write_inputs(d, gt=np.stack([gt] * n), monos=np.stack([mo] * n), splits=[sp[:s] for s in cuts],
                 calls=[ca[ca < s] for s in cuts], cmd=[cd[:s + 1] for s in cuts],
                 pbwt=np.concatenate([R.pbwt(c, K, reverse=r)[0] for c in crefs for r in (False, True)]),
                 count0=np.zeros(sum(map(len, crefs)), np.int32), rows=np.array([len(c) for c in crefs]), K=K, P=P,
                 prephase=prephase)
    pi = np.fromfile(os.path.join(d, "params_i.bin"), np.int32)
    # short histories: the heaps reach over several paths' buffers
    pi[3], pi[5], pi[6], pi[8] = H, H // 2, H, 0
    pi.tofile(os.path.join(d, "params_i.bin"))
    # the emulator's own barriers store their (equal) thread count on every use
    (d / "supp").write_text("race:pair_barrier\n")
    r = subprocess.run([exe, str(d)], capture_output=True, text=True, timeout=900,
                       env=dict(os.environ, TSAN_OPTIONS=f"suppressions={d}/supp history_size=4 exitcode=66"))
    assert r.returncode in (0, 66), f"rc {r.returncode}: {r.stderr[-4000:]}"
    out = []
    for rep in r.stderr.split("WARNING: ThreadSanitizer: data race")[1:]:
        out.append(re.findall(r"#\d+ (?:eimp::)?(?:\(anonymous namespace\)::)?(\w+)[^\n]*beam_emu", rep))
    assert bool(out) == (r.returncode == 66), r.stderr[-4000:]
    return out


def test_heaps_after_the_last_copies(emu_exe, tmp_path):
    """The constraint heaps are filled only when no path is being copied."""
    got = reports(emu_exe, tmp_path, 16, True, range(20, 30))
    assert not [s for s in got if any(f.startswith(("heap_", "constraint_heaps", "hswap")) for f in s)], got


@pytest.mark.parametrize("prephase,cuts", [(False, range(40, 43)), (True, range(24, 26))])
def test_free_slots_read_before_they_change(emu_exe, tmp_path, prephase, cuts):
    """The free-slot mask: every lane has read it before a lane stores it."""
    got = reports(emu_exe, tmp_path, 16, prephase, cuts)
    assert not [s for s in got if "beam_apply_hap" in s], got


@pytest.mark.parametrize("P,H,cuts", [(16, 8, range(24, 28)), (4, 2, range(30, 34)), (128, 30, range(44, 46))])
def test_nothing_reported(emu_exe, tmp_path, P, H, cuts):
    """Small and wide beams (more than 32 paths), a ring as long as the history
    (whose entry 0 is rescaled twice) and a longer one."""
    assert reports(emu_exe, tmp_path, P, True, cuts, H) == []
