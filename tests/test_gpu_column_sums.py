"""Column sums that finish in the kernel that adds them (csrc/elementwise.cu): one chunk of
rows, the first sizes with several, and columns no vector divides; the bias gradient of
dlb_fc_weight_gradient against float64."""
import ctypes

import numpy as np
import pytest

from dlb200 import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cols", [4, 10, 132, 257])
@pytest.mark.parametrize("rows", [1, 7, 64, 255, 256, 257, 3000])
def test_bias_gradient(gpu_ctx, rows, cols):
    ctx, rng = gpu_ctx, np.random.default_rng(rows + cols)
    d = rng.standard_normal((rows, cols), dtype=np.float32)
    x = np.ones((rows, 8), np.float32)
    start = rng.standard_normal(cols).astype(np.float32)
    dd, xd, dw, db = ctx.array(d), ctx.array(x), ctx.empty((cols, 8)), ctx.array(start)
    for accumulate, want in ((1, start + d.sum(0, dtype=np.float64)), (0, d.sum(0, dtype=np.float64))):
        check(ctx.L.dlb_fc_weight_gradient(ctx.h, dd.ptr, None, xd.ptr, None, dw.ptr, db.ptr, rows, 8, cols, accumulate))
        assert ctx.sync() == 0
        assert np.abs(db.get() - want).max() <= 3e-7 * np.sqrt(rows) * 4 + 3e-7


@pytest.mark.parametrize("rows,cols", [(7, 4), (200, 132), (3000, 256)])
def test_bias_gradient_of_an_unaligned_error(gpu_ctx, rows, cols):
    """An error tensor that starts one float past a 16-byte boundary."""
    ctx, rng = gpu_ctx, np.random.default_rng(rows)
    d = rng.standard_normal((rows, cols), dtype=np.float32)
    x = rng.standard_normal((rows, 8), dtype=np.float32)
    room = ctx.array(np.concatenate([np.zeros(1, np.float32), d.ravel()]))
    xd, dw, db = ctx.array(x), ctx.empty((cols, 8)), ctx.empty(cols)
    check(ctx.L.dlb_fc_weight_gradient(ctx.h, ctypes.c_void_p(room.ptr.value + 4), None, xd.ptr, None, dw.ptr, db.ptr, rows, 8, cols, 0))
    assert ctx.sync() == 0
    assert np.abs(db.get() - d.sum(0, dtype=np.float64)).max() <= 3e-7 * np.sqrt(rows) * 4 + 3e-7
    assert np.abs(dw.get() - d.T.astype(np.float64) @ x).max() <= 3e-6 * np.sqrt(rows) * 3
