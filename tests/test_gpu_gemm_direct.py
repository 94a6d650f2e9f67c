"""Products formed from the fp32 tensors by the tensor-core kernel that splits its
operands itself (csrc/gemm_direct.cu) and by the CUDA-core kernel for small ones
(csrc/gemm_small.cu): every size and pitch the plane kernels do not take, against the
float64 product, line by line."""
import numpy as np
import pytest

import util
from dlb200 import check

pytestmark = pytest.mark.gpu

# rows, n_in, n_out: edges of the 32 x 32 and 128 x 128 tiles and of the 128- and 64-deep
# chunks, one chunk, several CTAs per tile, more tiles than SMs, lines of odd and even
# pitch; the second line by the direct kernel (shallow large outputs, long thin sums).
SHAPES = [(1, 1, 1), (3, 65, 2), (127, 63, 129), (128, 64, 128), (129, 127, 130), (16, 784, 10), (1, 784, 256),
          (333, 617, 203), (200, 513, 1027), (1000, 66, 1001), (77, 2050, 77), (1700, 129, 1601), (31, 255, 33), (32, 256, 32), (1025, 127, 31),
          (1305, 23, 2213), (1001, 5, 2825), (951, 7735, 65), (130, 9001, 127)]


def _products(ctx, x, w, d, bias=None, start=None):
    """forward (+ bias), input gradient, weight gradient (added to `start`)."""
    L, (B, I), O = ctx.L, x.shape, w.shape[0]
    xd, wd, dd = (ctx.array(a) for a in (x, w, d))
    bd = ctx.array(bias) if bias is not None else None
    z, dx = ctx.empty((B, O)), ctx.empty((B, I))
    dw = ctx.array(start) if start is not None else ctx.empty((O, I))
    check(L.dlb_fc_forward(ctx.h, xd.ptr, None, wd.ptr, None, bd.ptr if bd else None, z.ptr, B, I, O))
    check(L.dlb_fc_backward_input(ctx.h, dd.ptr, None, wd.ptr, None, dx.ptr, B, I, O))
    check(L.dlb_fc_weight_gradient(ctx.h, dd.ptr, None, xd.ptr, None, dw.ptr, None, B, I, O, int(start is not None)))
    assert ctx.sync() == 0
    return z.get(), dx.get(), dw.get()


def _lines(got, want):
    return max(util.rowwise_rel_l2(got, want), util.rowwise_rel_l2(got.T, want.T))


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_products_of_any_size(gpu_ctx, shape):
    B, I, O = shape
    rng = np.random.default_rng(B + I + O)
    x, w, d = (rng.standard_normal(s, dtype=np.float32) for s in ((B, I), (O, I), (B, O)))
    bias, start = rng.standard_normal(O, dtype=np.float32), rng.standard_normal((O, I), dtype=np.float32)
    x64, w64, d64 = (a.astype(np.float64) for a in (x, w, d))
    got = _products(gpu_ctx, x, w, d, bias, start)
    for g, t, size in zip(got, (x64 @ w64.T + bias, d64 @ w64, d64.T @ x64 + start), (I, O, B)):
        # relative to the terms' size: single elements may cancel
        assert np.abs(g - t).max() <= 3e-6 * np.sqrt(size) * 3
        assert util.rel_l2(g, t) <= 1e-6


def test_lines_of_very_different_size(gpu_ctx):
    """Scales are per line and chunk: lines spread over 2^-20 .. 2^20 keep their own
    accuracy and no product is computed a second time."""
    rng = np.random.default_rng(2)
    x, w, d = (rng.standard_normal(s, dtype=np.float32) for s in ((150, 301), (203, 301), (150, 203)))
    for a in (x, w, d):
        a *= np.exp2(rng.uniform(-20, 20, a.shape[0])).astype(np.float32)[:, None]
    x64, w64, d64 = (a.astype(np.float64) for a in (x, w, d))
    before = gpu_ctx.guard_counters()
    z, dx, dw = _products(gpu_ctx, x, w, d)
    assert gpu_ctx.guard_counters() == before
    assert _lines(z, x64 @ w64.T) <= 1e-6
    assert util.rowwise_rel_l2(dx, d64 @ w64) <= 1e-6
    assert util.rel_l2(dw, d64.T @ x64) <= 1e-6


@pytest.mark.parametrize("value", [np.float32(2.0 ** 120), np.float32(np.inf), np.float32(np.nan), np.float32(1e-40)])
def test_values_the_halves_cannot_hold(gpu_ctx, value):
    rng = np.random.default_rng(3)
    x, w, d = (rng.standard_normal(s, dtype=np.float32) for s in ((140, 201), (150, 201), (140, 150)))
    x[131, 77] = value
    with np.errstate(all="ignore"):
        z, _, dw = _products(gpu_ctx, x, w, d)
        for got, want in ((z, x.astype(np.float64) @ w.T.astype(np.float64)), (dw, d.T.astype(np.float64) @ x.astype(np.float64))):
            finite = np.isfinite(want) & (np.abs(want) < 3e38)
            assert np.array_equal(np.isnan(got), np.isnan(want))
            assert np.array_equal(np.isfinite(got), finite)
            assert util.rel_l2(got[finite], want[finite]) <= 1e-6


B_SEED = 11
# Sizes at which gemm_direct.cu forms the product (the sizes above it leaves to other
# kernels): which product of the layer, one CTA and clusters per tile, operands contiguous
# along k and along the free dimension.
DIRECT = [((1000, 66, 1001), 0), ((1000, 66, 1001), 1), ((1000, 66, 1001), 2), ((951, 7735, 65), 0), ((951, 65, 7735), 1),
          ((7735, 65, 951), 2), ((2048, 256, 256), 1)]


def _direct_only(ctx, shape, which, x, w, d):
    """Product `which` of the layer, which must be gemm_direct_kernel's, and the guard's
    counters that it moved."""
    before, guard = ctx.product_counts(), ctx.guard_counters()
    L, (B, I, O) = ctx.L, shape
    xd, wd, dd = (ctx.array(a) for a in (x, w, d))
    out = ctx.empty(((B, O), (B, I), (O, I))[which])
    call = ((L.dlb_fc_forward, xd.ptr, None, wd.ptr, None, None, out.ptr, B, I, O),
            (L.dlb_fc_backward_input, dd.ptr, None, wd.ptr, None, out.ptr, B, I, O),
            (L.dlb_fc_weight_gradient, dd.ptr, None, xd.ptr, None, out.ptr, None, B, I, O, 0))[which]
    check(call[0](ctx.h, *call[1:]))
    assert ctx.sync() == 0
    assert {k for k, n in ctx.product_counts().items() if n != before[k]} == {"direct"}
    assert ctx.guard_counters() == guard
    return out.get()


def _exact(which, x, w, d):
    """The product and the largest error of an element.  S, the larger of the sum's own size
    and of sqrt(sum a^2 b^2), that of a sum whose signs are random: 22-bit operands move it
    by 2^-22 S at most in the mean square (five of that: 2^-20 S); the tensor core cuts
    off, 12 times in a chunk of 64 k, less than 2^-23 S; fp32 additions one by one move
    it by 0.3 2^-24 sqrt(k) S in the mean square."""
    x, w, d = (a.astype(np.float64) for a in (x, w, d))
    a, b = ((x, w.T), (d, w), (d.T, x))[which]
    exact = a @ b
    size = np.maximum(np.sqrt((a * a) @ (b * b)), np.abs(exact))
    return exact, size * (2.0 ** -20 + 12 * 2.0 ** -23 + 5 * 0.3 * 2.0 ** -24 * np.sqrt(a.shape[1]))


@pytest.mark.parametrize("shape,which", DIRECT)
def test_direct_kernel_lines_of_very_different_size(gpu_ctx, shape, which):
    """A scale per line and chunk: lines spread over 2^-20 .. 2^20 keep their own accuracy,
    where every row of the output is fed by one line of an operand."""
    rng, (B, I, O) = np.random.default_rng(B_SEED + which), shape
    x, w, d = (rng.standard_normal(s, dtype=np.float32) for s in ((B, I), (O, I), (B, O)))
    # of the two operands' free lines: rows of x and w; rows of d, columns of w; columns of d and x
    spread = lambda n: np.exp2(rng.uniform(-20, 20, n)).astype(np.float32)  # noqa: E731
    if which == 0:
        x, w = x * spread(B)[:, None], w * spread(O)[:, None]
    elif which == 1:
        d, w = d * spread(B)[:, None], w * spread(I)
    else:
        d, x = d * spread(O), x * spread(I)
    got, (want, bound) = _direct_only(gpu_ctx, shape, which, x, w, d), _exact(which, x, w, d)
    assert np.all(np.abs(got - want) <= bound)


@pytest.mark.parametrize("value", [2.0 ** 120, np.inf, np.nan, 1e-40])
@pytest.mark.parametrize("shape,which", DIRECT)
def test_direct_kernel_values_the_halves_cannot_hold(gpu_ctx, shape, which, value):
    """The tile of such a value is formed in fp32, by all CTAs of its cluster."""
    rng, (B, I, O) = np.random.default_rng(B_SEED + which), shape
    x, w, d = (rng.standard_normal(s, dtype=np.float32) for s in ((B, I), (O, I), (B, O)))
    (x, d, d)[which][B - 3, (I, O, O)[which] - 2] = np.float32(value)
    with np.errstate(all="ignore"):
        got, (want, bound) = _direct_only(gpu_ctx, shape, which, x, w, d), _exact(which, x, w, d)
        finite = np.isfinite(want) & (np.abs(want) < 3e38)
        assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isfinite(got), finite)
        assert np.all(np.abs(got - want)[finite] <= bound[finite])
