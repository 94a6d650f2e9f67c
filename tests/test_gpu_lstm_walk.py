"""The one-launch walk of an LSTM layer over time (csrc/lstm_walk.cu) at the edges of
its layouts: one CTA and clusters of 2 to 8, blocks that do not divide over them,
ragged groups of examples, one time step, odd and even numbers of cells, and more
cells than a warp has lanes (step by step); against the CPU restatement."""
import pytest

import configs
import dlb200
import fc_lstm
import util
from test_gpu_lstm import _check, _random_parameters

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,seq_w,blocks,cells", [
    (1, 3, 13, 3), (5, 1, 13, 3), (5, 2, 13, 2), (300, 4, 60, 2), (40, 3, 7, 4), (9, 3, 30, 5), (4, 3, 2, 33),
    (300, 2, 20, 1), (9, 3, 250, 1), (16, 3, 99, 4), (150, 3, 128, 2), (20, 2, 200, 2)])
def test_walk_matches_restatement(gpu_ctx, rows, seq_w, blocks, cells):
    cfg = configs.lstm_stack(n_in=24, blocks=blocks, cells=cells, depth=2, n_out=blocks * cells + 3, seq_w=seq_w,
                             batch=rows)
    X, Y = configs.synthetic_batch(cfg)
    p0 = _random_parameters(cfg)
    want = util.trace(util.build(fc_lstm.LstmOracleModel(), cfg, params=p0), cfg, 1, X, Y)
    got = util.trace(util.build(dlb200.Model(gpu_ctx), cfg, params=p0), cfg, 1, X, Y)
    assert gpu_ctx.sync() == 0
    _check(got, want, cfg)


# Sizes at which the plan takes each form (rows per warp x chunks of 128 k in registers, or
# weights in shared memory) with few and with many examples per cluster: forward / backward.
@pytest.mark.parametrize("rows,blocks,cells", [
    (5, 150, 2),   # 6 x 3 / 3 x 6
    (5, 200, 1),   # 10 x 2 / 2 x 10
    (16, 250, 1),  # shared memory / 2 x 10, two examples
    (16, 150, 2),  # shared memory / 3 x 6, two examples
    (40, 60, 3),   # 3 x 3, four examples / 3 x 3, two
    (200, 30, 3),  # 3 x 3, eight examples / 3 x 3, four
    (200, 99, 1),  # shared memory, eight examples / 2 x 5, eight
    (64, 128, 1),  # 5 x 2, five examples / 2 x 5
    (40, 150, 1),  # 5 x 2 / 2 x 5, four examples
    (150, 99, 1),  # shared memory, five examples / 2 x 5, five
])
def test_forms_of_the_walk(gpu_ctx, rows, blocks, cells):
    launches = []
    for seq_w in (2, 4):
        cfg = configs.lstm_stack(n_in=24, blocks=blocks, cells=cells, depth=1, n_out=blocks * cells + 3, seq_w=seq_w,
                                 batch=rows)
        X, Y = configs.synthetic_batch(cfg)
        p0 = _random_parameters(cfg)
        want = util.trace(util.build(fc_lstm.LstmOracleModel(), cfg, params=p0), cfg, 1, X, Y)
        model = util.build(dlb200.Model(gpu_ctx), cfg, params=p0)
        _check(util.trace(model, cfg, 1, X, Y), want, cfg)
        before = gpu_ctx.launch_count()
        model.forward_pass(rows, X)
        model.compute_error(rows, Y)
        model.backward_pass(rows)
        assert gpu_ctx.sync() == 0
        launches.append(gpu_ctx.launch_count() - before)
    # one launch per direction walks over all time steps
    assert launches[1] - launches[0] <= 1
