"""The update of all weight matrices in one launch (optimizer_matrices): more matrices than
one launch takes, of unequal shapes, against the update per vector that the TF32 form
runs, on the same gradients."""
import numpy as np
import pytest

import configs
import dlb200
import fc_step
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


# (AdaMax with decay: the reference has no AdaMax, and the restatement no decay for it)
@pytest.mark.parametrize("optimizer,decay", [(r, d) for d in (0.0, 1e-2) for r in (
    OPTIMIZER.ADAM, OPTIMIZER.AMSGRAD, OPTIMIZER.ADABOUND, OPTIMIZER.AMSBOUND, OPTIMIZER.NOSADAM)] + [(OPTIMIZER.ADAMAX, 0.0)])
def test_matrices_against_restatement(gpu_ctx, optimizer, decay):
    """Three updates of unequal matrices on given gradients, by the launch that takes them all:
    parameters and moments against the CPU restatement's, and the planes that the launch
    wrote through the forward pass that reads them."""
    cfg = configs.deep_brn_mlp(264, 512, 3, 384, 512, af=ACTIVATION.ISRLU, optimizer=optimizer, dropout=None, norm=False)
    X, Y = configs.synthetic_batch(cfg)
    mod = util.build(dlb200.Model(gpu_ctx), cfg, seed=0)
    p0 = mod.get_array("parameters")
    ora = util.build(fc_step.OracleModel(), cfg, params=p0)
    mod.train_begin(512)
    mod.train_step(512, X, Y)  # the weights' scales are predicted from here on
    mod.set_array("parameters", p0)
    moments = ["first_moment", "second_moment"]
    if optimizer in (OPTIMIZER.AMSGRAD, OPTIMIZER.AMSBOUND):
        moments.append("second_moment_hat")
    for name in moments:
        mod.set_array(name, np.zeros_like(p0))
    mod.set_hparam("optimizer_time_step", 0.0)
    mod.set_hparam("adam_previous_beta2", 0.0)
    rng = np.random.default_rng(1)
    for m in (mod, ora):
        m.set_weight_decay(decay)
    for _ in range(3):
        g = rng.standard_normal(p0.size).astype(np.float32)
        mod.forward_pass(512, X)  # planes of the weights as they are
        for m in (mod, ora):
            m.set_array("derivatives", g)
            m.update_weights(512, 512)
    mod.forward_pass(512, X)
    assert gpu_ctx.sync() == 0
    for name in ["parameters"] + moments:
        assert util.rel_max(mod.get_array(name), ora.get_array(name)) <= 2e-6, name
    ora.train_begin(512)
    ora.set_array("parameters", mod.get_array("parameters"))
    ora.forward_pass(512, X)
    last = len(cfg["layers"]) - 1
    assert util.rel_l2(mod.get_layer_outputs(last, 512), ora.get_layer_outputs(last, 512)) <= 1e-5
