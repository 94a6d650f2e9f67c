"""Forward products that keep their order of summation (csrc/gemm_ordered.cu): bit for bit
the CUDA-core kernel's results, at edges of the 64 x 64 tile and the 32-deep slab and up to
as many tiles as SMs."""
import numpy as np
import pytest

import configs
import dlb200
import util
from dlb200 import check
from enums import ACTIVATION

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,n_in,n_out", [(64, 129, 64), (70, 133, 65), (333, 617, 1203), (500, 333, 333), (65, 2049, 127)])
def test_same_bits_as_sums_in_ascending_k(gpu_ctx, rows, n_in, n_out):
    ctx, rng = gpu_ctx, np.random.default_rng(rows)
    x, w = rng.standard_normal((rows, n_in), dtype=np.float32), rng.standard_normal((n_out, n_in), dtype=np.float32)
    b = rng.standard_normal(n_out).astype(np.float32)
    xd, wd, bd, z = ctx.array(x), ctx.array(w), ctx.array(b), [ctx.empty((rows, n_out)) for _ in range(2)]
    try:
        for on in (0, 1):
            ctx.set_tensor_core(bool(on))
            check(ctx.L.dlb_fc_forward(ctx.h, xd.ptr, None, wd.ptr, None, bd.ptr, z[on].ptr, rows, n_in, n_out))
    finally:
        ctx.set_tensor_core(True)
    assert ctx.sync() == 0
    got = z[1].get()
    assert np.abs(got - (x.astype(np.float64) @ w.T + b)).max() <= 2e-6 * n_in ** 0.5 * 12
    if rows * n_out >= 128 * 128 and n_in < 2000:
        assert np.array_equal(got, z[0].get())


@pytest.mark.parametrize("af,norm,training,width,rows,kept", [
    (ACTIVATION.ELU, False, True, 1203, 333, True), (ACTIVATION.SELU, True, True, 1203, 333, True),
    (ACTIVATION.RELU, False, True, 1203, 333, True), (ACTIVATION.LEAKY_RELU, True, True, 1203, 333, True),
    # no derivative is taken, or none that jumps
    (ACTIVATION.ELU, False, False, 1203, 333, False), (ACTIVATION.SELU, True, False, 1203, 333, False),
    (ACTIVATION.ISRLU, False, True, 1203, 333, False), (ACTIVATION.ISRLU, True, True, 1203, 333, False),
    # shallower sums on planes would be less accurate than ascending ones
    (ACTIVATION.ELU, False, False, 617, 333, True), (ACTIVATION.ELU, False, False, 715, 333, False),
    # beyond what it may cost; a width TMA can address
    (ACTIVATION.ELU, False, True, 1203, 64, False), (ACTIVATION.ELU, False, True, 1203, 512, False),
    (ACTIVATION.ELU, False, True, 1200, 64, False), (ACTIVATION.ELU, False, True, 1200, 333, False)])
def test_forward_passes_that_keep_the_order(gpu_ctx, af, norm, training, width, rows, kept):
    cfg = configs.deep_brn_mlp(width, width, 2, 26, rows, af=af, dropout=None, norm=norm)
    X, _ = configs.synthetic_batch(cfg)
    model = util.build(dlb200.Model(gpu_ctx), cfg, seed=0)
    model.train_begin(rows)
    model.set_propagation(int(training))
    before = gpu_ctx.product_counts()
    model.forward_pass(rows, X)
    assert gpu_ctx.sync() == 0
    taken = {k: n - before[k] for k, n in gpu_ctx.product_counts().items()}
    # (the output layer of 26 is the small kernel's)
    assert taken["ordered"] == (2 if kept else 0) and sum(taken.values()) - taken["fresh_planes"] == 3
