"""GPU parity of the reference PBWT, the match search and the dosages against
the oracle on both sides of every size at which the build or the search takes
another form: four words of the order at a time from 16,384 haplotypes,
orders in an SM's shared memory up to some 33,200 (passes over the whole GPU
above), 16-bit intervals and rows through shared memory up to 65,536 (wide
intervals, rows in place above), blocks up to 262,144 (one CTA's walk above).
Site counts off a multiple of 16 and of 64, with and without sites past the
last block's first 16, searched in two parts."""
import numpy as np
import pytest

from eimp_b200.bits import W, pack_rows, unpack_rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,M", [(16382, 277), (16384, 277), (33236, 277), (33238, 277), (40000, 138), (65536, 277),
                                 (65538, 277), (262144, 85), (262146, 85)])
def test_against_oracle(ctx, K, M):
    from eimp_b200.engine import PBWTImputer
    from oracle import restate as R
    if not R.available():
        pytest.skip("oracle library not built")
    rng = np.random.default_rng(K + M)
    F, nt = 60, 4
    founders = rng.random((F, M)) < rng.choice([0.02, 0.3, 0.5], M)
    n = K + 2 * nt
    h = np.empty((n, M), np.uint8)
    src = rng.integers(0, F, n)
    for m in range(M):
        sw = np.flatnonzero(rng.random(n) < 0.02)
        src[sw] = rng.integers(0, F, len(sw))
        h[:, m] = founders[src, m]
    h ^= (rng.random(h.shape, dtype=np.float32) < 0.003).astype(np.uint8)
    if M > 200:
        h[:K, 64:128] = h[0, 64:128]   # a block that all agree in
    sm = pack_rows(np.ascontiguousarray(h[:K].T), W(K))
    th = h[K:]
    gt = np.where(rng.random((nt, M)) < 0.03, 3, th[0::2] + th[1::2]).astype(np.uint8)
    ph = pack_rows(th, W(M))
    typed = np.arange(0, M, dtype=np.int64)
    af = (h[:K].mean(axis=0)).astype(np.float32)
    imp = PBWTImputer(ctx, sm, af, typed, sm, K)
    imp.prepareImputation(ph, gt)
    compr, ap = imp.refpbwt()
    rc, rc0, rap = R.pbwt(sm, K, absperm=True)
    np.testing.assert_array_equal(ap.reshape(rap.shape), rap)
    np.testing.assert_array_equal(compr.reshape(rc.shape), rc)
    bits, dos = imp.impute_window(0, M)
    for t in range(2 * nt):
        miss = np.flatnonzero(gt[t // 2] == 3).astype(np.int64)
        om = R.smmatches(rc, rc0, M, K, ph[t], miss)
        np.testing.assert_array_equal(imp.matches(t).astype(np.int64), om)
        ob, od, sel = R.impute(om, rap, sm, typed, af, K, miss, ph[t])
        sel = sel.astype(bool)
        assert sel.sum() == len(miss)
        np.testing.assert_array_equal(dos[t][sel], od[sel])
        np.testing.assert_array_equal(unpack_rows(bits[t], M)[sel], unpack_rows(ob, M)[sel])
