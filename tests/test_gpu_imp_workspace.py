"""The device memory a context's first match search takes: global pools for the
lists that outgrow shared memory, one for each part a haplotype's sites can be
searched in."""
import numpy as np
import pytest

from eimp_b200.bits import W, pack_rows

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,errors", [(240, 0), (3000, 1)])
def test_first_search_of_one_part(M, errors):
    """240 sites are one part, and with set-maximal errors any number is."""
    import torch
    from eimp_b200.engine import Context, PBWTImputer
    rng = np.random.default_rng(M)
    K, nt = 512, 32
    h = (rng.random((8, M)) < 0.3)[rng.integers(0, 8, K + 2 * nt)].astype(np.uint8)
    h ^= (rng.random(h.shape) < 0.01).astype(np.uint8)
    sm = pack_rows(np.ascontiguousarray(h[:K].T), W(K))
    ctx = Context(0)
    imp = PBWTImputer(ctx, sm, np.full(M, 0.3, np.float32), np.arange(M), sm, K, setmaxerrors=errors)
    ctx.synchronize()
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    imp.prepareImputation(pack_rows(h[K:], W(M)), (h[K::2] + h[K + 1::2]).astype(np.uint8))
    taken = (before - torch.cuda.mem_get_info()[0]) / 2 ** 20
    ctx.close()
    # 64 haplotypes: a pool each of 4,096 entries in two buffers, at most 30
    # bytes an entry, is 7.5 MB (eight each, up to 256, are 23 to 30 MB); their
    # match buffers, genotypes and haplotypes are 1.2 MB at most; two megabytes a
    # buffer are the allocator's granularity
    assert taken <= 7.5 + 1.2 + 6
