"""Calls captured into CUDA graphs on parameters that the library has not seen before, and replayed after it has dropped them from
its caches."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import lstm_lib as ll
from rx_met_b200 import _cabi_lstm as L
from rx_met_b200 import gru_interface_binding as gru
from test_lstm_gpu import mod, torch_args

pytestmark = pytest.mark.gpu


def lstm_step(H, abits, seed):
    """Training forward and QAT backward of one LSTM layer as a function without arguments."""
    T, B, I = 5, 3, 12
    cfg = L.mixed_config(8, abits)
    p = ll.problem(T, B, I, H, seed=seed, wscale=float(1.0 / np.sqrt(H)))
    _, box = ll.calibrate("orc", cfg, p, np.stack([p["x"] * 0.8]))
    m, args = mod(), torch_args(p)
    bundle = m._params_to_bundle(box)
    g = [torch.ones(shape, device="cuda") for shape in ((T, B, H), (B, H), (B, H))]
    order = ("input", "weight_ih", "weight_hh", "bias_ih", "bias_hh", "h_0", "c_0")

    def run():
        out, hn, cn, ck, _ = m.lstm_forward_quantized(*args, False, bundle, "pedantic", False, True)
        qm, qk = ck["quantized_master"], ck["master_clamp_masks"]
        values = [ck["values"][n] for n in ("gate_outputs", "cell_states", "cell_tanh_outputs", "hidden_outputs")]
        grads = m.lstm_backward_qat([qm[n] for n in order], False, bundle, values, *g, [qk[n] for n in order],
                                    [ck["clamp_masks"][n] for n in L.TRACE_VALUES])
        return [out, hn, cn, *grads]
    return run


def gru_step(H, abits, seed):
    T, B, I = 5, 3, 12
    gen = torch.Generator().manual_seed(seed)
    rand = lambda *shape: (torch.rand(shape, generator=gen) - 0.5).cuda()  # noqa: E731
    W, R, bw, br, x, dh = rand(I, 3 * H), rand(H, 3 * H) * 0.2, rand(3 * H), rand(3 * H), rand(T, B, I), rand(T + 1, B, H)
    ranges = gru.GRUQuantizationRanges(H)
    gru.forward_calibrate(True, T, B, I, H, W, R, bw, br, x, None, "minmax", None, ranges)
    cfg = gru.OperatorQuantConfig()
    for name in ("x", "h", "weight_ih_linear", "weight_hh_linear"):
        setattr(cfg, f"{name}_", abits)
    params = gru.calculate_gru_quantitative_parameters(ranges, cfg)

    def run():
        out = gru.forward_quant_int_storage(True, T, B, I, H, W, R, bw, br, x, None, params)
        return [out[0], *gru.backward_quant_int_storage(T, B, I, H, *out[2:7], dh, out[0], out[1], params, *out[7:])]
    return run


@pytest.mark.parametrize("step,H,abits", [(lstm_step, 32, 8), (lstm_step, 96, 16), (lstm_step, 200, 8), (gru_step, 32, 8), (gru_step, 96, 16)],
                         ids=lambda v: v if isinstance(v, int) else v.__name__)
def test_first_use_of_parameters_inside_a_capture(step, H, abits):
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        step(H, abits, 1)()   # kernels and workspaces, on other parameters
    stream.synchronize()
    run = step(H, abits, 2)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        captured = run()
    graph.replay()
    torch.cuda.synchronize()
    want = [t.clone() for t in run()]
    for k, (a, b) in enumerate(zip(captured, want)):
        assert torch.equal(a, b), k
    # more parameter sets than the library keeps: the graph still reads its own
    for seed in range(3, 73):
        step(4, abits, seed)()
    spill = [torch.full((1 << 20,), 0x7f, dtype=torch.uint8, device="cuda") for _ in range(64)]
    for t in captured:
        t.zero_()
    graph.replay()
    torch.cuda.synchronize()
    del spill
    for k, (a, b) in enumerate(zip(captured, want)):
        assert torch.equal(a, b), k
