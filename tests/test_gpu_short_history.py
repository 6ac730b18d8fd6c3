"""Phasing with history sizes as long as the probability ring, on the GPU against
the oracle: a full path's oldest and newest ring entries are one, and the
rescaling takes it twice (HaplotypePath.cpp:224-258)."""
import numpy as np
import pytest

from conftest import golden_path

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prephase", [False, True])
@pytest.mark.parametrize("H", [2, 4, 8, 16, 32, 128])
def test_against_oracle(ctx, H, prephase):
    from eimp_b200.engine import PhaseParams, Phaser
    from oracle import restate as R
    if not R.available():
        pytest.skip("oracle library not built")
    g = np.load(golden_path("golden_tiny.npz"))
    hm, sm, cm = g["hapmajor_typed"], g["sitemajor_typed"], g["cm_typed"]
    o = dict(hsize=H, hsize_fast=H, delta=H // 2, delta_fast=0, doPrePhasing=prephase)
    got = Phaser(ctx, hm, sm, cm).phase(PhaseParams(K=64, beamwidth=16, **o), g["gt"])
    want = R.phase_many(g["gt"], hm, sm, cm, R.params_c(K=64, beamwidth=16, **o), 4)
    for a, b in zip(got[:4], want):
        np.testing.assert_array_equal(a, b)
