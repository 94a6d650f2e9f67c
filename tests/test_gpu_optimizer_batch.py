"""The update of all weight matrices in one launch (optimizer_matrices): more matrices than
one launch takes, of unequal shapes, against the update per vector that the TF32 form
runs, on the same gradients."""
import numpy as np
import pytest

import configs
import dlb200
import util
from enums import ACTIVATION, OPTIMIZER

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("optimizer", [OPTIMIZER.ADAM, OPTIMIZER.AMSBOUND])
def test_many_matrices(gpu_ctx, optimizer):
    cfg = configs.deep_brn_mlp(256, 512, 34, 384, 512, af=ACTIVATION.ISRLU, optimizer=optimizer, dropout=None, norm=False)
    X, Y = configs.synthetic_batch(cfg)
    after = {}
    try:
        for kind in (1, 0):
            gpu_ctx.set_gemm_kind(kind)
            model = util.build(dlb200.Model(gpu_ctx), cfg, seed=0)
            p0 = model.get_array("parameters")
            for _ in range(2):  # the second step's scales are predicted: all matrices in a launch
                model.set_array("parameters", p0)
                model.train_step(cfg["batch"], X, Y)
            # A gradient of the test's own, so that the two forms differ in the update only.
            rng = np.random.default_rng(0)
            hat = ("second_moment_hat",) if optimizer == OPTIMIZER.AMSBOUND else ()
            for name in ("first_moment", "second_moment") + hat:
                model.set_array(name, np.zeros_like(p0))
            model.set_hparam("optimizer_time_step", 0.0)
            model.set_array("parameters", p0)
            model.forward_pass(cfg["batch"], X)
            model.set_array("derivatives", rng.standard_normal(p0.size).astype(np.float32))
            model.update_weights(cfg["batch"], cfg["batch"])
            assert gpu_ctx.sync() == 0
            after[kind] = model.get_array("parameters")
            assert not model.get_array("derivatives").any()
    finally:
        gpu_ctx.set_gemm_kind(1)
    assert np.abs(after[1] - p0).min() > 0
    assert util.rel_max(after[1], after[0]) <= 1e-6
