"""Work that users of this framework run, as timed cases.

A case is one pass through the public entry points: the quantized GRU and LSTM forward (inference and training),
their QAT backward, calibration, the preallocated training engines and the learned-grid quantize-dequantize.
``listed()`` names fixed cases, ``draw()`` gives further ones of the same ranges.

Quantization parameters come from ranges that are written down here (the widths that standard normal inputs and
uniform initial weights give), not from a calibration pass, so that a case depends on its seed alone.
"""
import json
import math

import torch

from rx_met_b200 import _cabi, affine_qdq
from rx_met_b200 import _quant_lstm as lstm
from rx_met_b200 import gru_interface_binding as gru
from rx_met_b200.lstm_quant_params_io import canonical_float32
from rx_met_b200.qat import GruQatStep
from rx_met_b200.stacked_qat import StackedGruQat

DEVICE = "cuda"
LEARNING_RATE = 1e-3
LSTM_POINTS = ("weight_ih_linear", "weight_hh_linear", "gate_inputs", "gate_outputs", "cell_states",
               "cell_tanh_outputs", "hidden_outputs")
LSTM_MASTERS = ("input", "weight_ih", "weight_hh", "bias_ih", "bias_hh", "h_0", "c_0")
SAVED_POINTS = ("gate_outputs", "cell_states", "cell_tanh_outputs", "hidden_outputs")


def listed():
    return [
        # one utterance of a keyword spotter (98 frames of 40 features), answered as soon as it is there
        dict(name="gru_infer_one", kind="gru_infer", T=98, B=1, I=40, H=64, bits=8),
        # the same network over a batch: evaluation of a quantized model
        dict(name="gru_infer_batch", kind="gru_infer", T=98, B=32, I=40, H=64, bits=8),
        # min/max calibration of one batch of it
        dict(name="gru_calibrate", kind="gru_calibrate", T=98, B=32, I=40, H=64),
        # QAT through the call-by-call interface, at sizes that no tile divides
        dict(name="gru_train_ragged", kind="gru_train", T=61, B=45, I=29, H=100, bits=8),
        # QAT of a keyword spotter through the preallocated engine, one graph a step
        dict(name="gru_step", kind="gru_step", T=100, B=256, I=40, H=128, graph=True),
        # QAT of a stack of three bidirectional layers with 16-bit activations and a classifier
        dict(name="gru_body_step", kind="gru_body", T=100, B=128, I=40, H=256, layers=3, classes=12, graph=True),
        # a bidirectional layer with 16-bit activations over a batch
        dict(name="lstm_infer_bi", kind="lstm_infer", T=200, B=128, I=80, H=128, wbits=8, abits=16, directions=2),
        # one long sequence through a wide layer with 4-bit weights: latency
        dict(name="lstm_infer_one", kind="lstm_infer", T=1000, B=1, I=256, H=512, wbits=4, abits=16, directions=1),
        # the same layer at the batch of an offline job: throughput
        dict(name="lstm_infer_large", kind="lstm_infer", T=1000, B=4096, I=256, H=512, wbits=4, abits=16, directions=1),
        # QAT of a narrow 8-bit layer
        dict(name="lstm_train_a8", kind="lstm_train", T=100, B=256, I=40, H=128, wbits=8, abits=8),
        # QAT of the wide layer
        dict(name="lstm_train_wide", kind="lstm_train", T=1000, B=256, I=256, H=512, wbits=4, abits=16),
        # fake-quantized weight matrix with a trained grid per output row, forward and backward
        dict(name="qdq_weight", kind="qdq", rows=4096, cols=4096, grid="row", block=0),
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _width(rng, low, high):
    """A layer width: two of three are multiples of 32, as networks mostly have them, the others any number."""
    n = _log(rng, low, high)
    return n if rng.random() < 1 / 3 else min(high, max(32, (n + 16) // 32 * 32))


def draw(rng):
    kind = rng.choice(("gru_infer", "gru_calibrate", "gru_train", "gru_step", "gru_body", "lstm_infer", "lstm_train", "qdq"))
    if kind == "gru_infer":
        bits = rng.choice((8, 8, 16))
        return dict(kind=kind, T=_log(rng, 10, 400), B=_log(rng, 1, 1024), I=_width(rng, 8, 128), H=_width(rng, 16, 256), bits=bits)
    if kind == "gru_calibrate":
        return dict(kind=kind, T=_log(rng, 20, 200), B=_log(rng, 4, 256), I=_width(rng, 8, 128), H=_width(rng, 16, 256))
    if kind == "gru_train":
        bits = rng.choice((8, 8, 16))
        return dict(kind=kind, T=_log(rng, 20, 200), B=_log(rng, 8, 512), I=_width(rng, 8, 128), H=_width(rng, 16, 256), bits=bits)
    if kind == "gru_step":
        return dict(kind=kind, T=_log(rng, 40, 200), B=_log(rng, 16, 512), I=_width(rng, 8, 128), H=_width(rng, 32, 128),
                    graph=rng.random() < 0.7)
    if kind == "gru_body":
        return dict(kind=kind, T=_log(rng, 40, 150), B=_log(rng, 16, 256), I=_width(rng, 20, 80), H=rng.choice((64, 128, 192, 256)),
                    layers=rng.choice((2, 3)), classes=rng.randint(5, 40), graph=rng.random() < 0.7)
    if kind == "lstm_infer":
        wbits, abits, high = rng.choice(((8, 8, 128), (8, 16, 256), (4, 16, 512), (4, 16, 512)))
        big = high == 512
        return dict(kind=kind, T=_log(rng, 50, 1000 if big else 300), B=_log(rng, 1, 2048), I=_width(rng, 16, 256 if big else 128),
                    H=_width(rng, 256 if big else 32, high), wbits=wbits, abits=abits, directions=1 if big else rng.randint(1, 2))
    if kind == "lstm_train":
        wbits, abits, high = rng.choice(((8, 8, 128), (8, 16, 256), (4, 16, 512), (4, 16, 512)))
        big = high == 512
        return dict(kind=kind, T=_log(rng, 40, 500 if big else 200), B=_log(rng, 8, 256), I=_width(rng, 16, 256 if big else 128),
                    H=_width(rng, 256 if big else 32, high), wbits=wbits, abits=abits)
    grid = rng.choice(("tensor", "row", "column", "block"))
    block = 64 if grid == "block" else 0
    cols = _log(rng, 64, 8192)
    return dict(kind=kind, rows=_log(rng, 32, 16384), cols=(cols + 63) // 64 * 64 if block else cols, grid=grid, block=block)


# ---- inputs and parameters ---------------------------------------------------------------------------------------

def _normal(gen, *shape):
    return torch.randn(shape, generator=gen, device=DEVICE)


def _weights(gen, H, *shapes):
    """U(-1/sqrt(H), 1/sqrt(H)), as recurrent layers are initialised."""
    return [(torch.rand(s, generator=gen, device=DEVICE) * 2 - 1) / H ** 0.5 for s in shapes]


def _sigmoid(v):
    return 1 / (1 + math.exp(-v))


def _gru_config(bits):
    """8-bit symmetric weights per channel; activations of `bits` bits, asymmetric."""
    cfg = gru.OperatorQuantConfig()
    for name in _cabi.OP_NAMES:
        if name not in ("W", "R", "bw", "br"):
            setattr(cfg, name + "_", bits)
            setattr(cfg, name + "_symmetric_", False)
    return cfg


def _gru_params(W, R, bw, br, input_std, cfg):
    """Parameters from the ranges of about four standard deviations of every point of the cell."""
    I, H = W.shape[0], R.shape[0]
    ranges = gru.GRUQuantizationRanges(H)
    ih = 4 * input_std * (I / (3 * H)) ** 0.5 + 1 / H ** 0.5
    hh = 0.9
    spans = {"x": (-4 * input_std, 4 * input_std), "h": (-0.95, 0.95), "Wx": (-ih, ih), "Rh": (-hh, hh),
             "mul_reset_hidden": (-hh, hh), "mul_new_contribution": (-0.8, 0.8), "mul_old_contribution": (-0.8, 0.8)}
    gate = (ih * ih + hh * hh) ** 0.5
    for name in ("update_gate", "reset_gate", "new_gate"):
        spans[name + "_input"] = (-gate, gate)
        spans[name + "_output"] = ((-math.tanh(gate), math.tanh(gate)) if name == "new_gate" else
                                   (_sigmoid(-gate), _sigmoid(gate)))
    for name, (low, high) in spans.items():
        setattr(ranges, "min_%s_" % name, low)
        setattr(ranges, "max_%s_" % name, high)
    for name, t in (("W", W), ("R", R), ("bw", bw[None]), ("br", br[None])):
        setattr(ranges, "min_%s_" % name, t.amin(0).tolist())
        setattr(ranges, "max_%s_" % name, t.amax(0).tolist())
    return gru.calculate_gru_quantitative_parameters(ranges, cfg)


def _lstm_bundle(weights, wbits, abits):
    """Parameter document of one direction: symmetric weights per channel, asymmetric activations."""
    w_ih, w_hh = weights[:2]
    I, H = w_ih.shape[1], w_hh.shape[1]
    ih, hh = 4 * (I / (3 * H)) ** 0.5 + 1 / H ** 0.5, 0.9
    gate = (ih * ih + hh * hh) ** 0.5
    spans = {"input": (-4, 4), "output": (-0.8, 0.8), "cell_state": (-2, 2), "weight_ih_linear": (-ih, ih),
             "weight_hh_linear": (-hh, hh), "cell_gate_output": (-math.tanh(gate), math.tanh(gate)),
             "cell_tanh_output": (-0.97, 0.97)}
    for name in ("input_gate", "forget_gate", "cell_gate", "output_gate"):
        spans[name + "_input"] = (-gate, gate)
        if name != "cell_gate":
            spans[name + "_output"] = (0.0, _sigmoid(gate))
    ops = {}
    for name, (low, high) in spans.items():
        unsigned = low == 0.0
        scale = float(torch.tensor((high - low) / (2 ** abits - 1)))
        bottom = 0 if unsigned else -2 ** (abits - 1)
        ops[name] = dict(bitwidth=abits, is_unsigned=unsigned, is_symmetric=False, granularity="per_tensor",
                         scales=[canonical_float32(scale)], zero_points=[bottom + round(-low / scale)])
    for name, t in zip(LSTM_MASTERS[1:5], weights):
        bits = wbits if t.dim() == 2 else abits
        top = t.abs().reshape(4 * H, -1).amax(1).clamp_min(1e-6) / (2 ** (bits - 1) - 1)
        ops[name] = dict(bitwidth=bits, is_unsigned=False, is_symmetric=True, granularity="per_channel",
                         scales=[canonical_float32(s) for s in top.tolist()], zero_points=[0] * (4 * H))
    return json.dumps(dict(schema_version=1, input_size=I, hidden_size=H, bias_enabled=True, scale_mode="affine", operators=ops))


# ---- one state of each kind --------------------------------------------------------------------------------------

def prepare(case, seed):
    gen = torch.Generator(device=DEVICE).manual_seed(seed)
    kind = case["kind"]
    if kind == "qdq":
        rows, cols = case["rows"], case["cols"]
        x = _normal(gen, rows, cols) * 0.05
        shape = {"tensor": (1,), "row": (rows, 1), "column": (cols,), "block": (rows, cols // 64)}[case["grid"]]
        scale = 0.2 / 127 * (0.8 + 0.4 * torch.rand(shape, generator=gen, device=DEVICE))
        return dict(case=case, x=x.requires_grad_(), scale=scale.requires_grad_(),
                    offset=torch.zeros(shape, device=DEVICE).requires_grad_(), grad=_normal(gen, rows, cols))
    T, B, I, H = (case[k] for k in "TBIH")
    s = dict(case=case, x=_normal(gen, T, B, I))
    if kind in ("gru_infer", "gru_calibrate", "gru_train"):
        s["w"] = _weights(gen, H, (I, 3 * H), (H, 3 * H), (3 * H,), (3 * H,))
        s["config"] = _gru_config(case.get("bits", 8))
        if kind != "gru_calibrate":
            s["params"] = _gru_params(*s["w"], 1.0, s["config"])
        if kind == "gru_train":
            s["dh"] = _normal(gen, T + 1, B, H)
    elif kind == "gru_step":
        config = _gru_config(8)
        s["engine"] = engine = GruQatStep(T, B, I, H, DEVICE, config, seed=seed)
        engine.set_params(_gru_params(engine.W, engine.R, engine.bw, engine.br, 1.0, config))
        s["target"] = _normal(gen, T, B, H)
        if case["graph"]:
            s["replay"] = engine.capture_step(s["x"], s["target"], LEARNING_RATE)[0]
    elif kind == "gru_body":
        config = _gru_config(16)
        s["engine"] = engine = StackedGruQat(T, B, I, H, case["layers"], case["classes"], DEVICE, config, seed=seed)
        s["x"] = s["x"].clamp_(-4, 4)
        for k, pair in enumerate(engine.dirs):
            for d in pair:
                d.set_params(_gru_params(d.W, d.R, d.bw, d.br, 0.25 if k else 1.0, config))
        s["labels"] = torch.randint(0, case["classes"], (B,), generator=gen, device=DEVICE)
        if case["graph"]:
            s["replay"] = engine.capture_step(s["x"], s["labels"], LEARNING_RATE)[0]
    else:
        directions = case.get("directions", 1)
        s["w"] = [_weights(gen, H, (4 * H, I), (4 * H, H), (4 * H,), (4 * H,)) for _ in range(directions)]
        s["bundle"] = [_lstm_bundle(w, case["wbits"], case["abits"]) for w in s["w"]]
        if directions == 2:
            s["x_reversed"] = s["x"].flip(0)
            s["side"] = torch.cuda.Stream()
        if kind == "lstm_train":
            s["grads"] = [_normal(gen, T, B, H), _normal(gen, B, H), _normal(gen, B, H)]
    return s


# ---- one pass ----------------------------------------------------------------------------------------------------

def run(s):
    return globals()["_run_" + s["case"]["kind"]](s)


def _dims(s):
    return [s["case"][k] for k in "TBIH"]


def _run_gru_infer(s):
    return gru.forward_quant_int_storage(False, *_dims(s), *s["w"], s["x"], None, s["params"])[:2]


def _run_gru_calibrate(s):
    T, B, I, H = _dims(s)
    ranges = gru.GRUQuantizationRanges(H)
    h, v = gru.forward_calibrate(False, T, B, I, H, *s["w"], s["x"], None, "minmax", s["config"], ranges)
    points = ("x", "h", "Wx", "Rh", "update_gate_input", "update_gate_output", "reset_gate_input", "reset_gate_output",
              "new_gate_input", "new_gate_output", "mul_reset_hidden", "mul_old_contribution", "mul_new_contribution")
    spans = torch.tensor([getattr(ranges, "%s_%s_" % (end, p)) for p in points for end in ("min", "max")])
    channels = torch.tensor([getattr(ranges, "%s_%s_" % (end, p)) for p in ("W", "R") for end in ("min", "max")])
    biases = torch.tensor([getattr(ranges, "%s_%s_" % (end, p)) for p in ("bw", "br") for end in ("min", "max")])
    return h, v, spans, channels, biases


def _run_gru_train(s):
    dims = _dims(s)
    saved = gru.forward_quant_int_storage(True, *dims, *s["w"], s["x"], None, s["params"])
    h, v, codes, masks = saved[0], saved[1], saved[2:7], saved[7:]
    grads = gru.backward_quant_int_storage(*dims, *codes, s["dh"], h, v, s["params"], *masks)
    return saved, grads


def _run_gru_step(s):
    engine = s["engine"]
    loss = s["replay"]() if s["case"]["graph"] else engine.step(s["x"], s["target"], LEARNING_RATE)
    return loss, engine.flat_w, engine.flat_g, engine.h, engine.dx


def _run_gru_body(s):
    engine = s["engine"]
    loss = s["replay"]() if s["case"]["graph"] else engine.step(s["x"], s["labels"], LEARNING_RATE)
    return loss, engine.flat_w, engine.flat_g, engine.y[-1]


def _run_lstm_infer(s):
    if s["case"]["directions"] == 1:
        return lstm.lstm_forward_quantized(s["x"], *s["w"][0], None, None, False, s["bundle"][0])[:3]
    main, side = torch.cuda.current_stream(), s["side"]   # the two directions do not wait for one another
    side.wait_stream(main)
    ahead = lstm.lstm_forward_quantized(s["x"], *s["w"][0], None, None, False, s["bundle"][0])[:3]
    with torch.cuda.stream(side):
        back = lstm.lstm_forward_quantized(s["x_reversed"], *s["w"][1], None, None, False, s["bundle"][1])[:3]
    main.wait_stream(side)
    return ahead, back


def _run_lstm_train(s):
    out, h_n, c_n, saved, _ = lstm.lstm_forward_quantized(s["x"], *s["w"][0], None, None, False, s["bundle"][0], "pedantic",
                                                          False, True)
    grads = lstm.lstm_backward_qat([saved["quantized_master"][n] for n in LSTM_MASTERS], False, s["bundle"][0],
                                   [saved["values"][n] for n in SAVED_POINTS], *s["grads"],
                                   [saved["master_clamp_masks"][n] for n in LSTM_MASTERS],
                                   [saved["clamp_masks"][n] for n in LSTM_POINTS])
    return out, h_n, c_n, saved, grads


def _run_qdq(s):
    block = [1, s["case"]["block"]] if s["case"]["block"] else None
    y = affine_qdq.quantize_dequantize(s["x"], s["scale"], s["offset"], -128, 127, block)
    return (y.detach(),) + torch.autograd.grad(y, (s["x"], s["scale"], s["offset"]), s["grad"])


# ---- what a pass cannot do without -------------------------------------------------------------------------------

def work(case):
    """Every input read once and every output written once, saved tensors included where the interface returns
    them; the products of the gates with the input and the hidden state (backward: twice those of the forward)."""
    kind = case["kind"]
    if kind == "qdq":
        n = case["rows"] * case["cols"]
        return dict(bytes=16 * n, flops=16 * n)
    T, B, I, H = (case[k] for k in "TBIH")
    rows = T * B
    if kind == "gru_body":
        inputs = [I] + [2 * H] * (case["layers"] - 1)
        return dict(bytes=rows * sum(2 * (4 * i + 4 * H) for i in inputs),
                    flops=rows * sum(2 * 18 * H * (i + H) for i in inputs))
    if kind.startswith("gru"):
        weights = 4 * 3 * H * (I + H + 2)
        forward = dict(bytes=rows * (4 * I + 20 * H) + weights, flops=rows * 6 * H * (I + H))
        if kind == "gru_step":    # input, target, gradient of the input, the output
            return dict(bytes=rows * (8 * I + 8 * H) + 3 * weights, flops=3 * forward["flops"])
        if kind == "gru_train":   # codes and clamp flags on top of the forward, then the gradients
            saved = rows * (5 * I + 13 * H) + 2 * weights
            return dict(bytes=forward["bytes"] + saved + rows * (4 * I + 4 * H) + weights, flops=3 * forward["flops"])
        return forward
    weights = 4 * 4 * H * (I + H + 2)
    forward, flops = rows * (4 * I + 4 * H) + weights, rows * 8 * H * (I + H)
    if kind == "lstm_infer":
        return dict(bytes=case["directions"] * forward, flops=case["directions"] * flops)
    saved = rows * 5 * (I + 4 * 4 * H + 3 * H) + 2 * weights
    return dict(bytes=forward + saved + rows * (4 * I + 4 * H) + weights, flops=3 * flops)


def tolerance(case):
    """Codes, and what is computed from codes alone, are the same in every correct implementation.  Gradients and the
    float forward are sums in float32."""
    if case["kind"] in ("gru_infer", "lstm_infer"):
        return "exact"
    if case["kind"] in ("gru_step", "gru_body"):
        return dict(rel=5e-5)    # weights that differ in their last bits can move a code of a later step
    return dict(rel=1e-5)
