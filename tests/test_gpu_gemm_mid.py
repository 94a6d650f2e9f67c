"""Products on fp16 planes with 256 x 128 tiles whose k range up to four pairs of SMs
share (csrc/gemm_mid.cu): one, two and four pieces, ragged edges of tile and
k-block, mn-contiguous operands whose extent is no multiple of 64."""
import numpy as np
import pytest

import util
from dlb200 import check

pytestmark = pytest.mark.gpu

# rows, n_in, n_out with planes: pitches are multiples of 8; 512^3: four pieces of k
# per tile, 2048 x 1024 x 1024: one, 1024^3: two.
SHAPES = [(256, 256, 256), (512, 512, 512), (1024, 1024, 1024), (2048, 1024, 1024), (264, 136, 520), (300, 1000, 520),
          (1000, 520, 264), (257, 2056, 256), (3000, 72, 1032)]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_products_on_kept_planes(gpu_ctx, shape):
    ctx, L, (B, I, O) = gpu_ctx, gpu_ctx.L, shape
    rng = np.random.default_rng(B + I + O)
    x, w, d = (rng.standard_normal(s, dtype=np.float32) for s in ((B, I), (O, I), (B, O)))
    bias, start = rng.standard_normal(O, dtype=np.float32), rng.standard_normal((O, I), dtype=np.float32)
    (xd, xp), (wd, wp), (dd, dp) = ((ctx.array(a), ctx.empty(a.shape)) for a in (x, w, d))
    for t, p, a in ((xd, xp, x), (wd, wp, w), (dd, dp, d)):
        check(L.dlb_split_planes_2d(ctx.h, t.ptr, p.ptr, *a.shape))
    bd = ctx.array(bias)
    x64, w64, d64 = (a.astype(np.float64) for a in (x, w, d))
    runs = []
    for fill in (7.5, -3.25):  # what the outputs held before does not matter
        z, dx = ctx.array(np.full((B, O), fill, np.float32)), ctx.array(np.full((B, I), fill, np.float32))
        dw = ctx.array(start)
        check(L.dlb_fc_forward(ctx.h, xd.ptr, xp.ptr, wd.ptr, wp.ptr, bd.ptr, z.ptr, B, I, O))
        check(L.dlb_fc_backward_input(ctx.h, dd.ptr, dp.ptr, wd.ptr, wp.ptr, dx.ptr, B, I, O))
        check(L.dlb_fc_weight_gradient(ctx.h, dd.ptr, dp.ptr, xd.ptr, xp.ptr, dw.ptr, None, B, I, O, 1))
        assert ctx.sync() == 0
        runs.append((z.get(), dx.get(), dw.get()))
    for a, b, t in zip(*runs, (x64 @ w64.T + bias, d64 @ w64, d64.T @ x64 + start)):
        assert np.array_equal(a, b)
        assert util.rel_l2(a, t) <= 2e-6
        assert util.rowwise_rel_l2(a, t) <= 1e-5
