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
