"""GPU parity: Qref haplotype sections long enough to be indexed on a thread of
their own (eimp_b200/csrc/api.cu: eimp_qref_decode)."""
import numpy as np
import pytest

from eimp_b200.bits import W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nvar", [4095, 4096, 6001])
def test_sections_indexed_beside_the_copy(ctx, nvar):
    """From 4,096 variants on the section is indexed while it is copied: the
    rows, and a section that ends early at its last and at its first variant."""
    from eimp_b200.engine import EimpError, decode_qref_haplotypes
    from oracle import restate as R
    rng = np.random.default_rng(nvar)
    rows = rng.integers(0, 2 ** 63, (nvar, W(200))).astype(np.uint64)
    rows[::3] = 0
    rows[:, 200 // 64] &= np.uint64((1 << (200 % 64)) - 1)
    rows[:, 200 // 64 + 1:] = 0
    sec = R.qref_section(rows)
    np.testing.assert_array_equal(decode_qref_haplotypes(ctx, sec, nvar, 100), rows)
    for n in (sec.size - 1, 7):
        with pytest.raises(EimpError, match="Failed reading haplotypes"):
            decode_qref_haplotypes(ctx, sec[:n], nvar, 100)
    np.testing.assert_array_equal(decode_qref_haplotypes(ctx, sec, nvar, 100), rows)
