"""Element-wise kernels that write the operand planes of what they produce
(quad_rows_kernel in csrc/elementwise.cu): edges of the column blocks and row chunks, the
first call (planes by a split) and the second (planes by the kernel); the values against
NumPy and the planes through the product that reads them."""
import ctypes as C

import numpy as np
import pytest

import dlb200
import fc_step
import util
from dlb200 import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("op", ["bernoulli", "inverted", "uout", "none", "residual", "shakedrop"])
@pytest.mark.parametrize("rows,n", [(515, 132), (1025, 260), (33, 2052)])
def test_values_and_planes(gpu_ctx, op, rows, n):
    ctx, L, rng = gpu_ctx, gpu_ctx.L, np.random.default_rng(rows + n)
    rnd = lambda *s: rng.standard_normal(s, dtype=np.float32)  # noqa: E731
    x, other, noise, flags = rnd(rows, n), rnd(rows, n), rnd(rows, n), (rng.random(rows) < 0.4).astype(np.uint8)
    mask = (rng.random(n) < 0.8).astype(np.uint8)
    w = rnd(2048, n)
    xd, nd, fd, md, wd = (ctx.array(a) for a in (x, noise, flags, mask, w))
    out, planes, wp, z = ctx.empty((rows, n)), ctx.empty((rows, n)), ctx.empty(w.shape), ctx.empty((rows, 2048))
    check(L.dlb_split_planes_2d(ctx.h, wd.ptr, wp.ptr, 2048, n))
    shaken = np.where(flags[:, None] == 1, noise, np.float32(1))
    kind = {"bernoulli": fc_step.DROPOUT_BERNOULLI, "inverted": fc_step.DROPOUT_BERNOULLI_INVERTED,
            "uout": fc_step.DROPOUT_UOUT, "none": fc_step.DROPOUT_NONE}
    for _ in range(2):
        if op == "residual":
            od = ctx.array(other)
            check(L.dlb_residual_forward(ctx.h, xd.ptr, od.ptr, fd.ptr, nd.ptr, out.ptr, planes.ptr, rows, n))
            want = x + other * shaken
        elif op == "shakedrop":
            check(L.dlb_shakedrop_backward(ctx.h, xd.ptr, fd.ptr, nd.ptr, out.ptr, planes.ptr, rows, n))
            want = x * shaken
        else:
            dp = dlb200.DropoutDesc(kind[op], 0.8, md.ptr, nd.ptr)
            check(L.dlb_activation_forward(ctx.h, xd.ptr, None, fc_step.AF_LEAKY_RELU, C.byref(dp), out.ptr, planes.ptr,
                                           rows, n))
            want = fc_step.apply_dropout(fc_step.af_fire(fc_step.AF_LEAKY_RELU, x), kind[op], 0.8, mask, noise)
        check(L.dlb_fc_forward(ctx.h, out.ptr, planes.ptr, wd.ptr, wp.ptr, None, z.ptr, rows, n, 2048))
        assert ctx.sync() == 0
        assert util.rel_max(out.get(), want) <= 1e-6
        assert util.rel_l2(z.get(), want.astype(np.float64) @ w.T.astype(np.float64)) <= 2e-6
