"""Which kernel forms a product (gemm() in csrc/ctx.cu), by the kernels' own estimates: the
sizes that the tests of each kernel rely on reach it, with and without kept planes.  A
constant of an estimate that moves shows here which kernel its tests no longer run."""
import pytest

from dlb200 import check

pytestmark = pytest.mark.gpu

FRESH, FRESH_PAIR = "mid+fresh_planes", "pair+fresh_planes"
# rows, n_in, n_out: forward, input gradient, weight gradient
WITHOUT_PLANES = {
    # test_gpu_gemm_direct.py: the small kernel's tiles and pieces of k, the direct
    # kernel's one and several CTAs per tile in each direction
    (1, 1, 1): ("small", "small", "small"),
    (129, 127, 130): ("ordered", "small", "small"),
    (16, 784, 10): ("small", "small", "small"),
    (77, 2050, 77): ("small", "small", "small"),
    (1000, 66, 1001): ("direct", "direct", "direct"),
    (1305, 23, 2213): ("direct", "small", "small"),
    (951, 7735, 65): ("direct", FRESH, FRESH),
    (951, 65, 7735): (FRESH_PAIR, "direct", FRESH),
    (7735, 65, 951): (FRESH_PAIR, FRESH, "direct"),
    (2048, 256, 256): ("direct", "direct", FRESH),
    # test_gpu_split_lines.py
    (1024, 1000, 2048): (FRESH, FRESH, FRESH),
    (1001, 1203, 1030): (FRESH, FRESH, FRESH),
    (2050, 513, 1100): (FRESH_PAIR, FRESH, FRESH),
    (640, 2600, 515): (FRESH, FRESH, FRESH),
    # test_gpu_gemm_ordered.py
    (64, 129, 64): ("ordered", "small", "small"),
    (333, 617, 1203): ("ordered", FRESH, FRESH),
    (500, 333, 333): ("ordered", "small", "small"),
}
WITH_PLANES = {
    # test_gpu_gemm_mid.py: one, two and four pieces of k; the error of a weight
    # gradient whose rows are no whole 128-byte columns gets planes of its own
    (256, 256, 256): ("mid", "mid", "mid"),
    (512, 512, 512): ("mid", "mid", "mid"),
    (1024, 1024, 1024): ("mid", "mid", "mid"),
    (2048, 1024, 1024): ("mid", "mid", "mid"),
    (264, 136, 520): ("mid", "small", "small"),
    (300, 1000, 520): ("mid", "mid", FRESH),
    (257, 2056, 256): ("mid", "mid", "mid"),
    (3000, 72, 1032): ("pair", "mid", FRESH),
    # the headline layers
    (4096, 4096, 4096): ("pair", "pair", "pair"),
}


def _way(ctx, product, *args):
    """The kernels that a product took."""
    before = ctx.product_counts()
    check(product(ctx.h, *args))
    return "+".join(k for k, n in ctx.product_counts().items() if n != before[k])


@pytest.mark.parametrize("shape,planes,want", [(s, False, w) for s, w in WITHOUT_PLANES.items()] +
                         [(s, True, w) for s, w in WITH_PLANES.items()])
def test_kernel_of_each_product(gpu_ctx, shape, planes, want):
    ctx, L, (B, I, O) = gpu_ctx, gpu_ctx.L, shape
    x, w, d = (ctx.zeros(s) for s in ((B, I), (O, I), (B, O)))
    z, dx, dw = (ctx.zeros(s) for s in ((B, O), (B, I), (O, I)))
    xp = wp = dp = None
    if planes:
        xp, wp, dp = (ctx.zeros(s) for s in ((B, I), (O, I), (B, O)))
        for t, p, s in ((x, xp, (B, I)), (w, wp, (O, I)), (d, dp, (B, O))):
            check(L.dlb_split_planes_2d(ctx.h, t.ptr, p.ptr, *s))
    at = lambda a: a.ptr if a else None  # noqa: E731
    got = (_way(ctx, L.dlb_fc_forward, x.ptr, at(xp), w.ptr, at(wp), None, z.ptr, B, I, O),
           _way(ctx, L.dlb_fc_backward_input, d.ptr, at(dp), w.ptr, at(wp), dx.ptr, B, I, O),
           _way(ctx, L.dlb_fc_weight_gradient, d.ptr, at(dp), x.ptr, at(xp), dw.ptr, None, B, I, O, 0))
    assert ctx.sync() == 0
    assert got == want
