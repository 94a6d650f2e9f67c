"""ShakeDrop's flags and factors drawn in one launch (shakedrop_kernel in csrc/noise.cu) at
widths that whole generator blocks do and do not divide, against a step with the host
restatement's draws."""
import pytest

import configs
import dlb200
import fc_residual
import philox
import util

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,rows", [(50, 37), (131, 9), (260, 70)])
def test_step_with_drawn_noise(gpu_ctx, width, rows):
    seed, step = (3 << 33) | 7, 5
    cfg = configs.residual_mlp(width=width, blocks=3, n_out=7, batch=rows, p_last=0.2)
    X, Y = configs.synthetic_batch(cfg)
    mod = util.build(dlb200.Model(gpu_ctx), cfg, seed=4)
    ora = util.build(fc_residual.ResidualOracleModel(), cfg, params=mod.get_array("parameters"))
    for li, p in configs.shakedrop_layers(cfg):
        draw = lambda lo, s: philox.uniform(rows * width, lo, 1, seed, 4 * li + s, step).reshape(rows, width)  # noqa: E731
        ora.set_shakedrop_noise(li, philox.bernoulli(rows, p, seed, 4 * li, step), draw(-1, 1), draw(0, 2))
    mod.draw_noise(rows, seed, step)
    out = []
    for m in (ora, mod):
        m.train_begin(rows)
        m.reset_loss()
        m.forward_pass(rows, X)
        m.compute_error(rows, Y)
        m.backward_pass(rows)
        m.update_derivatives(rows)
        m.merge_derivatives()
        out.append((m.get_loss(), m.get_array("derivatives")))
    assert gpu_ctx.sync() == 0
    assert abs(out[0][0] - out[1][0]) <= 1e-5 * abs(out[0][0])
    assert util.rel_l2(out[1][1], out[0][1]) <= 2e-5
