"""The beam kernel with history sizes that are powers of two, on the CPU under
the warp emulator against the oracle.  The probability ring has exactly as many
entries as the history then, so a full path's oldest entry, which its
rescaling reaches, lies where its newest does: that one is rescaled twice
(HaplotypePath.cpp:224-258), whichever lanes take the two."""
import os

import numpy as np
import pytest

from conftest import golden_path
from test_beam_warp_emulated import emu_exe, golden_inputs, run_emu, write_inputs  # noqa: F401


@pytest.mark.parametrize("H", [1, 2, 4, 8, 16, 32, 64, 128])
def test_ring_as_long_as_the_history(emu_exe, tmp_path, H):  # noqa: F811
    from oracle import restate as R
    if not R.available():
        pytest.skip("oracle library not built")
    g = np.load(golden_path("golden_tiny.npz"))
    K, P, delta = 64, 16, H // 2
    write_inputs(tmp_path, K=K, P=P, prephase=True, **golden_inputs(g, K))
    pi = np.fromfile(os.path.join(tmp_path, "params_i.bin"), np.int32)
    pi[3], pi[5], pi[6], pi[8] = H, delta, H, delta
    pi.tofile(os.path.join(tmp_path, "params_i.bin"))
    nt, M = g["gt"].shape
    mats, pats, dm, dp, tc, nc, st = run_emu(emu_exe, tmp_path, nt, M)
    assert not st.any()
    p = R.params_c(K=K, beamwidth=P, hsize=H, hsize_fast=H, delta=delta, delta_fast=delta, doPrePhasing=True)
    om, op, odm, odp = R.phase_many(g["gt"], g["hapmajor_typed"], g["sitemajor_typed"], g["cm_typed"], p, 4)
    np.testing.assert_array_equal(mats, om)
    np.testing.assert_array_equal(pats, op)
    np.testing.assert_array_equal(dm, odm)
    np.testing.assert_array_equal(dp, odp)
