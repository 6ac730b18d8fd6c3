"""The beam kernel as it is launched -- haplotype-path slots in shared memory,
several warps per target -- on the CPU under the warp emulator with the
sanitizers: fewer slots than paths, so that paths are copied between shared
memory and the arena, and more.  Against the reference's golden phasing and,
with the pre-phasing pass and a wide beam, the oracle; the persistent form
takes all targets with one set of slots."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import golden_path
from test_beam_warp_emulated import CSRC, EMU, golden_inputs, run_emu, write_inputs


@pytest.fixture(scope="module", params=[(1, 1), (5, 2), (3, 4), (60, 4)], ids=lambda p: f"slots{p[0]}-warps{p[1]}")
def emu_exe(request, tmp_path_factory):
    if shutil.which("g++") is None:
        pytest.skip("g++ not available")
    slots, warps = request.param
    d = tmp_path_factory.mktemp("beam_slots_emu")
    for f in ("common.cuh", "kernels.h"):
        shutil.copy(os.path.join(CSRC, f), d / f)
    src = open(os.path.join(CSRC, "beam.cu")).read()
    i, j = src.index("static size_t beam_smem("), src.rindex("}  // namespace eimp")
    src = src[:i] + src[j:]
    for old, new in [("extern __shared__ __align__(16) uint8_t smem_raw[];", "uint8_t *smem_raw = emu_smem_ptr;"),
                     ("a.NS = 0;", f"a.NS = {slots};"), ("a.NR = 0;", f"a.NR = {slots + 3};")]:
        assert src.count(old) == 1
        src = src.replace(old, new)
    (d / "beam_emu.cpp").write_text('#include "emu.h"\n' + src)
    main = open(os.path.join(EMU, "beam_main.cpp")).read()
    for old, new, n in [
            ("eimp::beam_canon_bytes(al.NH);", "eimp::beam_canon_bytes(al.NH) + eimp::beam_slot_bytes(al.NS, al.HMAX, al.NR) + "
             f"eimp::beam_term_bytes({warps});", 1),
            ("EmuWarp warp;", f"std::vector<EmuWarp> warps({warps}); EmuBarrier block; block.n = {32 * warps};", 2),
            ("l < 32;", f"l < {32 * warps};", 2), ("blockDim.x = 32;", f"blockDim.x = {32 * warps};", 2),
            ("emu_warp = &warp;", "emu_warp = &warps[l / 32]; emu_block = &block;", 2)]:
        assert main.count(old) == n
        main = main.replace(old, new)
    (d / "main.cpp").write_text(main)
    exe = d / "beam_emu"
    r = subprocess.run(["g++", "-std=c++20", "-O1", "-g", "-ffp-contract=off", "-fno-fast-math",
                        "-fsanitize=address,undefined", "-fno-sanitize-recover=undefined", "-I", EMU, "-I", str(d),
                        str(d / "main.cpp"), "-o", str(exe), "-lpthread"], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-4000:]
    return str(exe)


@pytest.mark.parametrize("K", [50, 200])
def test_slots(emu_exe, tmp_path, K):
    g = np.load(golden_path("golden_tiny.npz"))
    pre = f"K{K}_"
    write_inputs(tmp_path, K=K, P=16, prephase=False, **golden_inputs(g, K))
    nt, M = g["gt"].shape
    mats, pats, dm, dp, tc, nc, st = run_emu(emu_exe, tmp_path, nt, M, queue=True)
    assert not st.any()
    np.testing.assert_array_equal(mats, g[pre + "mat"])
    np.testing.assert_array_equal(pats, g[pre + "pat"])
    np.testing.assert_array_equal(dm, g[pre + "dos_mat"])
    np.testing.assert_array_equal(dp, g[pre + "dos_pat"])
    np.testing.assert_array_equal(tc, g[pre + "totalconf"])
    np.testing.assert_array_equal(nc, g[pre + "ncallsites"])


def test_wide_beam_and_prephasing(emu_exe, tmp_path):
    """Beams beyond 32 paths (the general code), and constraints."""
    from oracle import restate as R
    g = np.load(golden_path("golden_tiny.npz"))
    inp = golden_inputs(g, 200)
    inp = {k: (v[:3] if k not in ("pbwt", "count0", "rows") else v) for k, v in inp.items()}
    rows = int(g["K200_rows"][:3].sum())
    inp["rows"], inp["pbwt"], inp["count0"] = g["K200_rows"][:3], inp["pbwt"][:2 * rows], inp["count0"][:rows]
    write_inputs(tmp_path, K=200, P=128, prephase=True, **inp)
    M = inp["gt"].shape[1]
    mats, pats, dm, dp, tc, nc, st = run_emu(emu_exe, tmp_path, 3, M)
    assert not st.any()
    p = R.params_c(K=200, beamwidth=128, doPrePhasing=True)
    for t in range(3):
        om, op, odm, odp, otc, onc = R.phase(inp["gt"][t], g["hapmajor_typed"], g["sitemajor_typed"], g["cm_typed"], p)
        np.testing.assert_array_equal(mats[t], om)
        np.testing.assert_array_equal(pats[t], op)
        np.testing.assert_array_equal(dm[t], odm)
        np.testing.assert_array_equal(dp[t], odp)
        assert tc[t] == np.float32(otc) and nc[t] == onc
