"""GPU parity of the phasing with many conditioning haplotypes against the
oracle: the beam's ring of three PBWT row pairs up to K = 16,384 and of two
above, and at 38,000 with more targets than SMs no room for haplotype-path
slots in shared memory; a few of each batch's targets are compared."""
import numpy as np
import pytest

from eimp_b200.bits import W, pack_rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,nt,prephase", [(16384, 40, False), (16386, 40, True), (16386, 460, False),
                                           (38000, 460, True)])
def test_against_oracle(ctx, K, nt, prephase):
    from eimp_b200.engine import PhaseParams, Phaser
    from oracle import restate as R
    if not R.available():
        pytest.skip("oracle library not built")
    rng = np.random.default_rng(K + nt)
    N, M, F = K + 500, 150, 80
    founders = rng.random((F, M)) < rng.choice([0.05, 0.3, 0.5], M)
    n = N + 2 * nt
    h = np.empty((n, M), np.uint8)
    src = rng.integers(0, F, n)
    for m in range(M):
        sw = np.flatnonzero(rng.random(n) < 0.02)
        src[sw] = rng.integers(0, F, len(sw))
        h[:, m] = founders[src, m]
    h ^= (rng.random(h.shape, dtype=np.float32) < 0.003).astype(np.uint8)
    hm, sm = pack_rows(h[:N], W(M)), pack_rows(np.ascontiguousarray(h[:N].T), W(N))
    gt = (h[N::2] + h[N + 1::2]).astype(np.uint8)
    gt[rng.random(gt.shape) < 0.01] = 3
    cm = np.cumsum(rng.random(M) * 0.02).astype(np.float32)
    got = Phaser(ctx, hm, sm, cm).phase(PhaseParams(K=K, beamwidth=128, doPrePhasing=prephase), gt)
    some = np.unique(np.linspace(0, nt - 1, 8).astype(int))
    want = R.phase_many(np.ascontiguousarray(gt[some]), hm, sm, cm, R.params_c(K=K, beamwidth=128, doPrePhasing=prephase), 8)
    for a, b in zip(got[:4], want):
        np.testing.assert_array_equal(a[some], b)
