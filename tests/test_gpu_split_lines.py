"""Planes made for one product with a scale per line (split_lines_kernel in
csrc/planes.cu), at sizes where that is the shorter way: lines longer than a warp or a
CTA keeps in registers, rows and columns that no vector or tile divides, lines of
very different size, infinities and NaN; against the float64 product."""
import numpy as np
import pytest

import util
from test_gpu_gemm_direct import _lines, _products

pytestmark = pytest.mark.gpu

SHAPES = [(1024, 1000, 2048), (1001, 1203, 1030), (2050, 513, 1100), (640, 2600, 515), (1300, 1029, 777)]


@pytest.mark.parametrize("spread", [0, 20])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_products_on_fresh_planes(gpu_ctx, shape, spread):
    B, I, O = shape
    rng = np.random.default_rng(B + I + O)
    x, w, d = (rng.standard_normal(s, dtype=np.float32) for s in ((B, I), (O, I), (B, O)))
    for a in (x, w, d):
        a *= np.exp2(rng.uniform(-spread, spread, a.shape[0])).astype(np.float32)[:, None]
    bias, start = rng.standard_normal(O, dtype=np.float32), rng.standard_normal((O, I), dtype=np.float32)
    x64, w64, d64 = (a.astype(np.float64) for a in (x, w, d))
    before = gpu_ctx.guard_counters()
    z, dx, dw = _products(gpu_ctx, x, w, d, bias, start)
    assert gpu_ctx.guard_counters() == before
    assert util.rel_l2(z, x64 @ w64.T + bias) <= 1e-6 and util.rel_l2(dw, d64.T @ x64 + start) <= 1e-6
    z, dx, dw = _products(gpu_ctx, x, w, d)
    assert _lines(z, x64 @ w64.T) <= 1.5e-6
    assert util.rowwise_rel_l2(dx, d64 @ w64) <= 1.5e-6
    assert util.rel_l2(dw, d64.T @ x64) <= 1e-6


@pytest.mark.parametrize("value", [np.inf, np.nan, 2.0 ** 120])
def test_values_the_halves_cannot_hold(gpu_ctx, value):
    rng = np.random.default_rng(3)
    x, w, d = (rng.standard_normal(s, dtype=np.float32) for s in ((1024, 1000), (2048, 1000), (1024, 2048)))
    x[1000, 997] = np.float32(value)
    with np.errstate(all="ignore"):
        z, _, dw = _products(gpu_ctx, x, w, d)
        x64, w64, d64 = (a.astype(np.float64) for a in (x, w, d))
        for got, want in ((z, x64 @ w64.T), (dw, d64.T @ x64)):
            finite = np.isfinite(want) & (np.abs(want) < 3e38)
            assert np.array_equal(np.isnan(got), np.isnan(want)) and np.array_equal(np.isfinite(got), finite)
            assert util.rel_l2(got[finite], want[finite]) <= 1e-6
    x[1000, 997] = 1.0  # the flag is the launch's own
    before = gpu_ctx.guard_counters()
    z, _, _ = _products(gpu_ctx, x, w, d)
    assert gpu_ctx.guard_counters() == before and util.rel_l2(z, x.astype(np.float64) @ w64.T) <= 1e-6
