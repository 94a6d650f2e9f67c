"""Which tensors keep operand planes is decided per batch size (choose_planes in
csrc/model.cu): a model that goes back and forth between batches whose products read
planes and batches whose products do not, against the CPU restatement step by step."""
import numpy as np
import pytest

import configs
import dlb200
import fc_step
import util
from enums import ACTIVATION, OPTIMIZER

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("norm", [True, False], ids=["normalised", "plain"])
def test_batches_that_do_and_do_not_keep_planes(gpu_ctx, norm):
    # ISRLU: a continuous derivative
    cfg = configs.deep_brn_mlp(256, 512, 2, 256, 512, af=ACTIVATION.ISRLU, optimizer=OPTIMIZER.ADAM, dropout=None,
                               norm=norm)
    X, Y = configs.synthetic_batch(cfg)
    mod = util.build(dlb200.Model(gpu_ctx), cfg, seed=0)
    ora = util.build(fc_step.OracleModel(), cfg, params=mod.get_array("parameters"))
    for m in (mod, ora):
        m.train_begin(cfg["batch"])
    for rows in (512, 24, 512, 24, 24, 512):
        losses = []
        for m in (mod, ora):
            m.reset_loss()
            m.forward_pass(rows, X[:rows])
            m.compute_error(rows, Y[:rows])
            m.backward_pass(rows)
            m.update_derivatives(rows)
            m.merge_derivatives()
            m.update_weights(rows, rows)
            losses.append(m.get_loss())
        assert abs(losses[0] - losses[1]) <= 2e-5 * abs(losses[1]), rows
    assert gpu_ctx.sync() == 0
    assert util.rel_l2(mod.get_array("parameters"), ora.get_array("parameters")) <= 1e-4


@pytest.mark.parametrize("norm", [True, False], ids=["normalised", "plain"])
def test_a_change_of_rows_keeps_the_registrations(gpu_ctx, norm):
    """Batches of two sizes, both of which keep planes: after the first step at either, a
    step launches the same kernels whether the rows changed before it or not (a producer
    whose registration is dropped cannot write the planes itself), and the weights
    follow the restatement's."""
    cfg = configs.deep_brn_mlp(256, 512, 2, 256, 640, af=ACTIVATION.ISRLU, optimizer=OPTIMIZER.ADAM, dropout=None,
                               norm=norm)
    X, Y = configs.synthetic_batch(cfg)
    mod = util.build(dlb200.Model(gpu_ctx), cfg, seed=0)
    ora = util.build(fc_step.OracleModel(), cfg, params=mod.get_array("parameters"))
    sizes = (640, 640, 640, 512, 512, 512, 640, 512, 640, 512)
    launches = []
    for m in (mod, ora):
        m.train_begin(cfg["batch"])
        for rows in sizes:
            before = gpu_ctx.launch_count()
            m.train_step(rows, X[:rows], Y[:rows])
            launches.append(gpu_ctx.launch_count() - before)
    assert gpu_ctx.sync() == 0
    for rows in (640, 512):
        steps = [n for r, n in zip(sizes, launches) if r == rows]
        assert set(steps[1:]) == {steps[2]}
    assert util.rel_l2(mod.get_array("parameters"), ora.get_array("parameters")) <= 1e-4
