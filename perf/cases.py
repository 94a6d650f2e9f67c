"""Timed cases of the library: what a user's program has it do, through the calls
that such a program makes.

A case is a dict.  `kind` says what one pass of it is:

  train      `steps` training steps of a model, the loss of every step read where
             the loop reads it, and the weights brought to the host at the end,
             as before a checkpoint.  `feed` is how the batches come in:
               epoch    MiniBatch.train over a data set in host memory
               staged   stage_batch / train_step_staged, page-locked batches
               rows     the step entry points one by one (the reference's own loop)
               device   batches that are on the GPU already
  predict    an evaluation pass: outputs and loss of `rows` examples from host
             memory, normalization by the running averages
  layer      the three products of one fully connected layer on tensors the
             caller owns (the library keeps nothing between the calls)
  optimizer  one update of a flat vector of `n` parameters
"""
import ctypes
import math
import os
import sys

import torch

sys.path.insert(0, os.path.abspath("deep-learning_b200"))

import configs  # noqa: E402
import dlb200  # noqa: E402
from enums import ACTIVATION, LAYER, LAYER_DROPOUT, OPTIMIZER  # noqa: E402

AF = {"relu": ACTIVATION.RELU, "lrelu": ACTIVATION.LEAKY_RELU, "elu": ACTIVATION.ELU, "selu": ACTIVATION.SELU,
      "isrlu": ACTIVATION.ISRLU}
DROPOUT = {"none": None, "bernoulli": LAYER_DROPOUT.BERNOULLI, "inverted": LAYER_DROPOUT.BERNOULLI_INVERTED,
           "uout": LAYER_DROPOUT.UOUT}
RULE = {"adam": OPTIMIZER.ADAM, "amsgrad": OPTIMIZER.AMSGRAD, "adabound": OPTIMIZER.ADABOUND,
        "amsbound": OPTIMIZER.AMSBOUND, "nosadam": OPTIMIZER.NOSADAM, "adamax": OPTIMIZER.ADAMAX}
HYPER = dict(adam_learning_rate=1e-4, adam_beta1=0.9, adam_beta2=0.999, adam_epsilon=1e-8,
             learning_rate_final=0.1, learning_gamma=1e-3, adam_gamma=0.1)


def mlp(kind, feed, n_in, hidden, depth, n_out, rows, steps=1, **more):
    """A stack of `depth` hidden layers: batch renormalization or bias, softmax
    classes or linear outputs."""
    c = dict(kind=kind, net="mlp", feed=feed, n_in=n_in, hidden=hidden, depth=depth, n_out=n_out, rows=rows,
             steps=steps, norm=True, softmax=False, af="selu", dropout="bernoulli", rule="adam")
    c.update(more)
    return c


def listed():
    return [
        # One example through the 784-256-10 classifier: the smallest call of a
        # program that answers requests, all latency.
        dict(mlp("predict", "rows", 784, 256, 1, 10, 1, norm=False, softmax=True, af="lrelu", dropout="none"),
             name="predict_784-256-10_b1"),
        # The same classifier's evaluation over a test set of 10000 in one call.
        dict(mlp("predict", "rows", 784, 256, 1, 10, 10000, norm=False, softmax=True, af="lrelu", dropout="none"),
             name="predict_784-256-10_b10000"),
        # Its training: an epoch of shuffled mini-batches of 128, the last one
        # longer by the remainder.
        dict(mlp("train", "epoch", 784, 256, 1, 10, 128, 16, norm=False, softmax=True, af="lrelu", dropout="none"),
             name="epoch_784-256-10_b128"),
        # A classifier whose inputs, widths and classes are what the data gives:
        # no multiple of a tile or of an alignment anywhere.
        dict(mlp("train", "staged", 617, 1203, 3, 26, 333, 4, norm=False, softmax=True, af="elu", dropout="inverted"),
             name="odd_617-3x1203-26_b333"),
        # The reduced deep batch-renorm MLP, driven through the step entry points
        # as the reference's own loop drives its model.
        dict(mlp("train", "rows", 256, 1024, 4, 256, 1024, 4, rule="amsbound"), name="brn_256-4x1024-256_b1024"),
        # The headline workload, batches staged one step ahead.
        dict(mlp("train", "staged", 1024, 4096, 4, 1024, 4096, 8, rule="amsbound"),
             name="brn_1024-4x4096-1024_b4096"),
        # The same kind of stack with bias instead of normalization, data on the GPU.
        dict(mlp("train", "device", 1024, 2048, 4, 1024, 2048, 4, norm=False, af="relu", dropout="uout"),
             name="plain_1024-4x2048-1024_b2048"),
        # Residual blocks with ShakeDrop, softmax over 1000 classes.
        dict(kind="train", net="residual", feed="staged", hidden=1024, blocks=8, n_out=1000, rows=2048, steps=4,
             rule="adam", name="residual_8x1024-1000_b2048"),
        # IndRNN stack, back-propagation through time from the last step.
        dict(kind="train", net="indrnn", feed="device", n_in=512, hidden=1024, depth=4, n_out=512, seq_w=64, rows=256,
             steps=2, rule="adabound", name="indrnn_512-4x1024-512_T64_b256"),
        # LSTM layers (memory blocks of two cells), errors on every time step.
        dict(kind="train", net="lstm", feed="device", n_in=128, blocks=128, cells=2, depth=2, n_out=256, seq_w=32,
             rows=64, steps=1, rule="adam", name="lstm_128-2x128x2-256_T32_b64"),
        # One layer called product by product by a program with its own training loop.
        dict(kind="layer", rows=1024, n_in=1000, n_out=2048, name="layer_1000-2048_b1024"),
        # The update alone, on a vector whose gradient another program merged.
        dict(kind="optimizer", n=100_000_000, rule="amsbound", name="optimizer_amsbound_1e8"),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def width(lo, hi):
        # Hidden widths are mostly chosen by hand: multiples of 64 or of 8 more often than not.
        step = rng.choice((64, 64, 8, 1))
        return max(lo, size(lo, hi) // step * step)

    family = rng.choice(("predict", "classifier", "brn", "brn", "plain", "residual", "indrnn", "lstm", "layer",
                         "optimizer"))
    if family == "predict":
        return mlp("predict", "rows", size(16, 1024), width(64, 2048), rng.randint(1, 4), size(2, 1000), size(1, 10000),
                   norm=rng.random() < 0.5, softmax=True, af=rng.choice(sorted(AF)), dropout="none")
    if family == "classifier":
        return mlp("train", rng.choice(("epoch", "staged", "rows")), size(16, 1024), width(64, 2048), rng.randint(1, 4),
                   size(2, 1000), size(16, 1024), rng.randint(2, 8), norm=False, softmax=True,
                   af=rng.choice(sorted(AF)), dropout=rng.choice(("none", "inverted", "bernoulli")),
                   rule=rng.choice(sorted(RULE)))
    if family in ("brn", "plain"):
        norm = family == "brn"
        return mlp("train", rng.choice(("staged", "rows", "device")), size(64, 1024), width(256, 4096),
                   rng.randint(2, 4), size(64, 1024), size(128, 4096), rng.randint(2, 8), norm=norm,
                   af=rng.choice(sorted(AF)),
                   dropout=rng.choice(("none", "bernoulli", "inverted") if norm else ("none", "bernoulli", "uout")),
                   rule=rng.choice(sorted(RULE)))
    if family == "residual":
        return dict(kind="train", net="residual", feed=rng.choice(("staged", "device")), hidden=width(128, 2048),
                    blocks=rng.randint(2, 8), n_out=size(10, 1000), rows=size(64, 2048), steps=rng.randint(1, 4),
                    rule=rng.choice(("adam", "amsgrad")))
    if family == "indrnn":
        return dict(kind="train", net="indrnn", feed="device", n_in=size(16, 512), hidden=width(64, 1024),
                    depth=rng.randint(1, 4), n_out=size(4, 512), seq_w=size(8, 64), rows=size(16, 256),
                    steps=rng.randint(1, 2), rule=rng.choice(("adam", "adabound")))
    if family == "lstm":
        blocks, cells = size(8, 128), rng.randint(1, 2)
        return dict(kind="train", net="lstm", feed="device", n_in=size(8, 128), blocks=blocks, cells=cells,
                    depth=rng.randint(1, 2), n_out=blocks * cells + size(1, 64), seq_w=size(4, 32), rows=size(8, 64),
                    steps=rng.randint(1, 2), rule=rng.choice(("adam", "amsgrad")))
    if family == "layer":
        return dict(kind="layer", rows=size(64, 4096), n_in=width(64, 4096), n_out=width(64, 4096))
    return dict(kind="optimizer", n=size(1_000_000, 100_000_000), rule=rng.choice(sorted(RULE)))


def config_of(c):
    """The workload description of configs.py for a model case."""
    if c["net"] == "residual":
        cfg = configs.residual_mlp(c["hidden"], c["blocks"], c["n_out"], c["rows"])
    elif c["net"] == "indrnn":
        cfg = configs.indrnn_stack(c["n_in"], c["hidden"], c["depth"], c["n_out"], c["seq_w"], c["rows"])
    elif c["net"] == "lstm":
        cfg = configs.lstm_stack(c["n_in"], c["blocks"], c["cells"], c["depth"], c["n_out"], c["seq_w"], c["rows"])
    else:
        d = DROPOUT[c["dropout"]]
        keep = 0.1 if d == LAYER_DROPOUT.UOUT else 0.9
        cfg = configs.deep_brn_mlp(c["n_in"], c["hidden"], c["depth"], c["n_out"], c["rows"], af=AF[c["af"]],
                                   keep=keep, dropout=d, norm=c["norm"])
        if c["softmax"]:
            s = configs.mlp_softmax()
            cfg["layers"][-1]["af"] = ACTIVATION.SOFTMAX
            cfg.update(loss=s["loss"], inputs=s["inputs"], targets=s["targets"])
    cfg.update(optimizer=RULE[c["rule"]], hparams=HYPER)
    return cfg


def make_batch(cfg, rows, gen):
    """Inputs and targets of `rows` examples as page-locked host arrays."""
    T, n_in, n_out = cfg["seq_w"], configs.n_inputs(cfg), configs.n_outputs(cfg)
    draw_x = torch.rand if cfg["inputs"] == "uniform" else torch.randn
    x = draw_x((rows, T * n_in), generator=gen, device="cuda")
    if cfg["targets"] == "onehot":
        labels = torch.randint(n_out, (rows * T, 1), generator=gen, device="cuda")
        y = torch.zeros((rows * T, n_out), device="cuda").scatter_(1, labels, 1.0).reshape(rows, T * n_out)
    else:
        y = torch.randn((rows, T * n_out), generator=gen, device="cuda")
    return [torch.empty(t.shape, pin_memory=True).copy_(t).numpy() for t in (x, y)]


def prepare(case, seed):
    c = case
    gen = torch.Generator(device="cuda").manual_seed(seed)
    ctx = dlb200.Context(0)
    s = {"case": c, "ctx": ctx, "L": ctx.L}
    if c["kind"] == "layer":
        B, I, O = c["rows"], c["n_in"], c["n_out"]
        normal = lambda *shape: torch.randn(shape, generator=gen, device="cuda")  # noqa: E731
        s.update(X=normal(B, I), W=normal(O, I).mul_(I ** -0.5), bias=normal(O).mul_(0.1), delta=normal(B, O).div_(B))
        s.update(Z=torch.empty(B, O, device="cuda"), dX=torch.empty(B, I, device="cuda"),
                 dW=torch.empty(O, I, device="cuda"), db=torch.empty(O, device="cuda"))
        return s
    if c["kind"] == "optimizer":
        n = c["n"]
        s["p"] = torch.randn(n, generator=gen, device="cuda").mul_(0.02)
        s["merged"] = torch.randn(n, generator=gen, device="cuda").mul_(1e-3)
        s["g"] = torch.zeros(n, device="cuda")
        s["moments"] = [torch.zeros(n, device="cuda") for _ in range(3)]
        s["time_step"], s["nos"] = ctypes.c_float(0.0), ctypes.c_float(0.0)
        s["scalars"] = dlb200.OptimizerScalars()
        # learning rate, beta1, beta2, epsilon, gamma, final rate, bound gamma, bias correction
        s["hyper"] = (ctypes.c_float * 8)(1e-4, 0.9, 0.999, 1e-8, 0.1, 0.1, 1e-3, 1.0)
        return s
    cfg = config_of(c)
    m = configs.build_model(dlb200.Model(ctx), cfg)
    m.seed_weights(seed & 0x7fffffff)
    m.initialize_weights_with_glorot_uniform()
    s.update(model=m, cfg=cfg, seed=seed)
    if c["kind"] == "predict":
        m.set_propagation(0)
        s["X"], s["Y"] = make_batch(cfg, c["rows"], gen)
        return s
    m.draw_noise(c["rows"], seed, 0)
    n = m.size("total_parameters")
    s["weights"] = torch.empty(n, pin_memory=True).numpy()
    if c["feed"] == "epoch":
        # The last batch is longer than the others: the remainder of the data set.
        s["X"], s["Y"] = make_batch(cfg, c["rows"] * c["steps"] + c["rows"] // 4, gen)
        s["loop"] = dlb200.MiniBatch(m, s["X"], s["Y"], c["rows"], use_shuffle=True, seed=seed & 0x7fffffff)
    else:
        s["batches"] = [make_batch(cfg, c["rows"], gen) for _ in range(min(c["steps"], 2))]
        if c["feed"] == "device":
            s["batches"] = [[ctx.array(a) for a in b] for b in s["batches"]]
    return s


def ptr(t):
    return t.data_ptr()


def run(s):
    c = s["case"]
    if c["kind"] == "layer":
        L, h, B, I, O = s["L"], s["ctx"].h, c["rows"], c["n_in"], c["n_out"]
        X, W, delta = ptr(s["X"]), ptr(s["W"]), ptr(s["delta"])
        dlb200.check(L.dlb_fc_forward(h, X, None, W, None, ptr(s["bias"]), ptr(s["Z"]), B, I, O))
        dlb200.check(L.dlb_fc_backward_input(h, delta, None, W, None, ptr(s["dX"]), B, I, O))
        dlb200.check(L.dlb_fc_weight_gradient(h, delta, None, X, None, ptr(s["dW"]), ptr(s["db"]), B, I, O, 0))
        return [s["Z"], s["dX"], s["dW"], s["db"]]
    if c["kind"] == "optimizer":
        L, h, n, rule = s["L"], s["ctx"].h, c["n"], RULE[c["rule"]]
        first, second, hat = s["moments"]
        dlb200.check(L.dlb_memcpy_d2d(h, ptr(s["g"]), ptr(s["merged"]), 4 * n))
        dlb200.check(L.dlb_optimizer_prepare(rule, s["hyper"], s["time_step"], s["nos"], s["scalars"]))
        dlb200.check(L.dlb_optimizer_step(h, rule, s["scalars"], ptr(s["p"]), ptr(s["g"]), ptr(first), ptr(second),
                                          ptr(hat), None, n))
        return [s["p"], s["g"], first, second] + ([hat] if c["rule"].startswith("ams") else [])
    m, rows = s["model"], c["rows"]
    if c["kind"] == "predict":
        m.reset_loss()
        m.forward_pass(rows, s["X"])
        m.compute_loss(rows, s["Y"])
        return [m.get_layer_outputs(len(s["cfg"]["layers"]) - 1, rows), m.get_loss()]
    return [train(s, m, c, rows), weights_to_host(s, m)]


def train(s, m, c, rows):
    """`steps` training steps; the losses as the loop of this feed reads them."""
    if c["feed"] == "epoch":
        return [s["loop"].train()]
    steps, batches, losses = c["steps"], s["batches"], []
    batch = lambda k: batches[k % len(batches)]  # noqa: E731
    if c["feed"] == "staged":
        m.stage_batch(rows, *batch(0))
    for k in range(steps):
        # Dropout masks and ShakeDrop draws are new in every step of a pass.
        m.draw_noise(rows, s["seed"], k)
        if c["feed"] == "staged":
            if k + 1 < steps:
                m.stage_batch(rows, *batch(k + 1))
            losses.append(m.train_step_staged())
        elif c["feed"] == "device":
            m.train_step_device(rows, *batch(k))
        else:
            x, y = batch(k)
            m.reset_loss()
            m.forward_pass(rows, x)
            m.compute_error(rows, y)
            m.backward_pass(rows)
            m.update_derivatives(rows)
            m.merge_derivatives()
            m.update_weights(rows, rows)
            losses.append(m.get_loss())
    if c["feed"] == "device":
        losses.append(m.get_loss())  # with the data on the GPU the loop looks at the loss now and then
    return losses


def weights_to_host(s, m):
    w = s["weights"]
    dlb200.check(s["L"].dlb_model_get_array(m.h, b"parameters", w.ctypes.data, w.size), "get_array")
    return w


def matrices(cfg):
    """(fan-in, fan-out, the error goes to what is below) of every product's weights."""
    out, below = [], configs.n_inputs(cfg)
    for l in cfg["layers"][1:]:
        if l["type"] == LAYER.RESIDUAL:
            continue
        units = l["units"]
        if l["type"] == LAYER.LSTM:
            cells = l["units"] * l["cells"]
            gates = cells + 3 * l["units"]
            out += [(below, gates, bool(out)), (cells, gates, True)]
            units = cells
        else:
            out.append((below, units, bool(out)))
        below = units
    return out


def work(case):
    c = case
    if c["kind"] == "layer":
        B, I, O = c["rows"], c["n_in"], c["n_out"]
        return {"bytes": 4.0 * (2 * B * I + 2 * B * O + 2 * O * I + 2 * O), "flops": 6.0 * B * I * O}
    vectors = {"amsgrad": 3, "amsbound": 3}
    if c["kind"] == "optimizer":
        # merged gradient read and parameters and moments read and written, gradient cleared
        return {"bytes": 4.0 * c["n"] * (2 + 2 + 2 * vectors.get(c["rule"], 2)), "flops": 10.0 * c["n"]}
    cfg = config_of(c)
    T, mats = cfg["seq_w"], matrices(cfg)
    weights = sum(i * o for i, o, _ in mats)
    values = c["rows"] * T * (configs.n_inputs(cfg) + configs.n_outputs(cfg))
    if c["kind"] == "predict":
        out = c["rows"] * T * configs.n_outputs(cfg)
        return {"bytes": 4.0 * (values + weights + out), "flops": 2.0 * c["rows"] * T * weights}
    through = sum(i * o for i, o, down in mats if down)
    # Every step reads its batch.  Weights and moments are read and written every
    # step where they are larger than the 126 MB L2, else once a pass.  The
    # weights go to the host at the end.
    state = weights * (2 + 2 * vectors.get(c["rule"], 2))
    passes = c["steps"] if 2 * state > 126e6 else 1
    return {"bytes": 4.0 * (c["steps"] * values + passes * state + weights),
            "flops": 2.0 * c["steps"] * c["rows"] * T * (2 * weights + through)}


def tolerance(case):
    """Products and sums are fp32 on 22-bit operands: 1e-5 on what one pass of
    them puts out.  Weights after several Adam-type steps: 1e-4, and a few of
    them more, because a first step has the size of the learning rate whatever
    the gradient's, so that a gradient within rounding of zero (or whose
    pre-activation is, at a kink of the activation) moves its weight by up to
    twice that."""
    if case["kind"] == "optimizer":
        return {"rel": 1e-6, "max": 1e-4}
    if case["kind"] == "train":
        return {"rel": 1e-4, "max": 0.2}
    return {"rel": 1e-5, "max": 1e-3}
