"""eimp_kernel_launches counts every kernel a call launches: the builds of the
reference PBWT by blocks of sites (orders in an SM's shared memory, or passes
over the GPU above some 33,200 haplotypes) or by one CTA's walk, and the match
search in one part or several."""
import numpy as np
import pytest

from eimp_b200.bits import W, pack_rows

pytestmark = pytest.mark.gpu


def build(ctx, rng, K, M, errors=0):
    from eimp_b200.engine import PBWTImputer
    h = (rng.random((M, 1)) < 0.3) ^ (rng.random((M, K)) < 0.05)
    sm = pack_rows(h.astype(np.uint8), W(K))
    n = ctx.launches
    imp = PBWTImputer(ctx, sm, np.full(M, 0.3, np.float32), np.arange(M), sm, K, setmaxerrors=errors)
    return imp, h, ctx.launches - n


# transpose, segment map and fill; keys, ranks of blocks and of groups, orders of
# groups and of blocks, orders inside blocks; without full blocks before the
# last no ranks; with two blocks one group; up to 16 sites the walk.  Wide: keys,
# ranks, 2 launches for every 6 bits of a rank and block, 9 x 2 inside blocks
@pytest.mark.parametrize("K,M,want", [(2000, 300, 9), (2000, 100, 8), (2000, 40, 6), (2000, 16, 4),
                                      (40000, 150, 3 + 2 + 2 * 3 * 2 + 2 * 3 * 3)])
def test_reference(K, M, want):
    from eimp_b200.engine import Context
    ctx = Context(0)
    _, _, n = build(ctx, np.random.default_rng(M), K, M)
    ctx.synchronize()
    ctx.close()
    assert n == want


# 600 sites of few haplotypes in several parts, which are joined; then the retry
@pytest.mark.parametrize("M,errors,want", [(100, 0, 2), (600, 0, 3), (600, 1, 2)])
def test_search(M, errors, want):
    from eimp_b200.engine import Context
    rng = np.random.default_rng(M)
    ctx = Context(0)
    imp, h, _ = build(ctx, rng, 500, M, errors)
    th = np.ascontiguousarray(h[:, :4].T).astype(np.uint8)
    n = ctx.launches
    imp.prepareImputation(pack_rows(th, W(M)), (th[0::2] + th[1::2]).astype(np.uint8))
    n = ctx.launches - n
    ctx.close()
    assert n == want
