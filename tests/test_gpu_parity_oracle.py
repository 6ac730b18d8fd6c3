"""GPU parity against the oracle restatement of two settings that are otherwise
checked against the reference-compiled oracle only, where its sources are
there: a haploid region of the 5,000-haplotype panel, and the full phase and
impute configuration (10,000 haplotypes x 100,000 sites, 5,000 typed,
K = 4,096, beam 128) on its first targets."""
import os

import numpy as np
import pytest

from eimp_b200.bits import W, pack_rows, transpose_bits, unpack_rows

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def oracle():
    from oracle import restate as R
    if not R.available():
        pytest.skip("oracle library not built")


def check_imputation(imp, bits, dos, compr, c0, ap, cols, panel, typed, hap, gt, rows):
    """Matches, and alleles and dosages where there is something to impute;
    cols: the panel column of each haplotype of the reference PBWT."""
    from oracle import restate as R
    M, Mref = len(typed), panel.nsites
    apc = cols[ap].astype(np.int32)
    for h in rows:
        miss = np.flatnonzero(gt[h // 2] == 3).astype(np.int64)
        om = R.smmatches(compr, c0, M, ap.shape[1], hap[h], miss)
        np.testing.assert_array_equal(imp.matches(int(h)).astype(np.int64), om)
        ob, od, sel = R.impute(om, apc, panel.sitemajor, typed, panel.af, panel.nhaps, miss, hap[h])
        sel = sel.astype(bool)
        assert sel.sum() == Mref - M + len(miss)
        np.testing.assert_array_equal(dos[h][sel], od[sel])
        np.testing.assert_array_equal(unpack_rows(bits[h], Mref)[sel], unpack_rows(ob, Mref)[sel])


def test_haploid_region(ctx):
    """Every third reference sample haploid, 5 of 16 targets haploid, K = 1,024
    and beam 64.  The oracle runs over the columns that exist."""
    from eimp_b200 import synth
    from eimp_b200.engine import PBWTImputer, PhaseParams, Phaser
    from oracle import restate as R
    panel, groups = synth.generate("cfg1")
    tg = groups[0]
    nt, nh, Mref = 16, panel.nhaps, panel.nsites
    ref_hap = (np.arange(nh // 2) % 3 == 1).astype(np.uint8)
    second = 2 * np.flatnonzero(ref_hap) + 1
    dense = unpack_rows(panel.hapmajor, Mref)
    dense[second] = dense[second - 1]
    hm_full = pack_rows(dense, W(Mref))
    panel = synth.Panel(nh, Mref, panel.pos, panel.cm, (dense.sum(axis=0) / nh).astype(np.float32), hm_full,
                        transpose_bits(hm_full, nh, Mref))
    tgt_hap = np.zeros(nt, np.uint8)
    tgt_hap[[0, 3, 7, 8, 15]] = 1
    gt = tg.gt[:nt].copy()
    for t in np.flatnonzero(tgt_hap):
        gt[t] = np.where(gt[t] == 3, 3, 2 * tg.truth[2 * t])
    hm, sm, cm = synth.typed_views(panel, tg.typed)
    M = len(tg.typed)
    cols = np.delete(np.arange(nh), second)
    hm_r = np.ascontiguousarray(hm[cols])
    sm_r = transpose_bits(hm_r, len(cols), M)
    ph = Phaser(ctx, hm, sm, cm)
    ph.setHaploidRef(ref_hap)
    ph.setHaploidTargets(tgt_hap)
    mats, pats, dm, dp, tc, nc = ph.phase(PhaseParams(K=1024, beamwidth=64), gt)
    ph.setHaploidTargets(None)
    dip = np.flatnonzero(tgt_hap == 0)
    om, op, odm, odp = R.phase_many(np.ascontiguousarray(gt[dip]), hm_r, sm_r, cm, R.params_c(K=1024, beamwidth=64),
                                    os.cpu_count() or 1)
    for a, b in ((mats, om), (pats, op), (dm, odm), (dp, odp)):
        np.testing.assert_array_equal(a[dip], b)
    hap = np.zeros((2 * nt, W(M)), np.uint64)
    hap[0::2], hap[1::2] = mats, pats
    imp = PBWTImputer(ctx, panel.sitemajor, panel.af, tg.typed, sm, nh, haploid_ref=ref_hap)
    assert imp.K == len(cols)
    imp.prepareImputation(hap, gt, haploid_targets=tgt_hap)
    bits, dos = imp.impute_window(0, Mref)
    # the imputation PBWT of a second haplotype whose column starts a word of the
    # reduced rows: the reference loses its bits (Datatypes.h:190-197)
    lost = (np.arange(len(cols)) % 64 == 0) & (cols % 2 == 1)
    assert lost.any()
    alleles = unpack_rows(sm_r, len(cols))
    alleles[:, lost] = 0
    compr, c0, ap = R.pbwt(pack_rows(alleles, W(len(cols))), len(cols), absperm=True)
    gc, ga = imp.refpbwt()
    np.testing.assert_array_equal(gc, compr)
    np.testing.assert_array_equal(ga, ap)
    rows = [h for h in range(2 * nt) if h % 2 == 0 or not tgt_hap[h // 2]]
    assert len(rows) == 27
    check_imputation(imp, bits, dos, compr, c0, ap, cols, panel, tg.typed, hap, gt, rows)


def test_full_configuration(ctx):
    from eimp_b200 import synth
    from eimp_b200.engine import PBWTImputer, PhaseParams, Phaser
    from oracle import restate as R
    panel, groups = synth.generate("cfg2")
    tg = groups[0]
    nt, K, beam = 24, 4096, 128
    gt = np.ascontiguousarray(tg.gt[:nt])
    hm, sm, cm = synth.typed_views(panel, tg.typed)
    M, Mref = len(tg.typed), panel.nsites
    mats, pats, dm, dp, tc, nc = Phaser(ctx, hm, sm, cm).phase(PhaseParams(K=K, beamwidth=beam), gt)
    om, op, odm, odp = R.phase_many(gt, hm, sm, cm, R.params_c(K=K, beamwidth=beam), os.cpu_count() or 1)
    for a, b in ((mats, om), (pats, op), (dm, odm), (dp, odp)):
        np.testing.assert_array_equal(a, b)
    hap = np.zeros((2 * nt, W(M)), np.uint64)
    hap[0::2], hap[1::2] = mats, pats
    imp = PBWTImputer(ctx, panel.sitemajor, panel.af, tg.typed, sm, panel.nhaps)
    imp.prepareImputation(hap, gt)
    bits, dos = imp.impute_window(0, Mref)
    compr, c0, ap = R.pbwt(sm, panel.nhaps, absperm=True)
    gc, ga = imp.refpbwt()
    np.testing.assert_array_equal(gc, compr)
    np.testing.assert_array_equal(ga, ap)
    check_imputation(imp, bits, dos, compr, c0, ap, np.arange(panel.nhaps), panel, tg.typed, hap, gt, range(2 * nt))
