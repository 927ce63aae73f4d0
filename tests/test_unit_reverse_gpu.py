"""The reverse recurrences with a thread per hidden unit (QAT backward up to 128 units): one, two and four rows of a CTA per copy of the weights with
the last CTA partly empty, two rows of a thread over more steps than the ring of operands has slots, against the CPU checkers."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

import gpu_lib as gl
import oracle_lib as ol
from test_gru_gpu import test_backward_quant as gru_backward_matches
from test_lstm_wide_gpu import test_wide_qat_backward as lstm_backward_matches

pytestmark = pytest.mark.gpu


# 516 inputs keep widths of 32 and 96 from padded copies
@pytest.mark.parametrize("T,B,I,H", [(6, 593, 8, 128), (9, 149, 8, 128), (7, 1185, 8, 64), (6, 595, 8, 64), (5, 2369, 516, 32), (6, 1185, 516, 32), (6, 593, 516, 96),
                                     (5, 149, 516, 96)])
def test_gru_rows(T, B, I, H):
    gru_backward_matches(gl, "w8a8", (T, B, I, H))


@pytest.mark.parametrize("T,B,I,H", [(6, 297, 8, 128), (9, 149, 8, 128), (7, 1185, 8, 64), (6, 595, 8, 64), (6, 2369, 8, 32), (6, 593, 8, 96)])
def test_lstm_rows(T, B, I, H):
    lstm_backward_matches(T, B, I, H, 8, 16)


@pytest.mark.parametrize("H", [64, 128])
def test_lstm_misaligned_weight_codes(monkeypatch, H):
    """Weight codes four bytes beside a 16-byte boundary, which the kernel's wide loads need."""
    import torch
    from test_lstm_gpu import mod
    m = mod()
    backward = m.lstm_backward_qat

    def shifted(masters, *rest):
        masters = list(masters)
        w = masters[2]
        masters[2] = torch.empty(w.numel() + 1, dtype=w.dtype, device="cuda")[1:].view(w.shape).copy_(w)
        return backward(masters, *rest)

    monkeypatch.setattr(m, "lstm_backward_qat", shifted)
    lstm_backward_matches(5, 9, 8, H, 8, 16)


@pytest.mark.parametrize("B,H", [(16, 32), (64, 32), (45, 64), (128, 64)])
def test_gru_error_of_narrow_layers(B, H):
    """Sums over the channels of a part in one truncating accumulator: dh0 after 60 steps stays as near to the checker's (64-bit sums) as where each
    gate had an accumulator of its own: 7.1e-8 then, 6.2e-8 now of its norm, limit 1.5e-7."""
    T, I = 60, 8
    cfg = ol.make_config(bits=8, symmetric=False)
    prob = ol.gru_problem(B + H, T, B, I, H, with_h0=True)
    ranges, params = ol.RangesBox(H), ol.ParamsBox(H, cfg)
    gl.forward_float(*prob, ranges=ranges)
    assert gl.cabi.load_library().rxmet_gru_params_from_ranges(C.byref(ranges.c), C.byref(cfg), C.byref(params.c)) == 0
    f = ol.forward_quant("orc", *prob, params, training=True)
    dh = np.zeros((T + 1, B, H), np.float32)
    dh[1:] = np.random.default_rng(H).standard_normal((T, B, H)).astype(np.float32)
    want = ol.backward_quant(f, dh, f["h"], f["v"], params, f["masks"])["dh0"].astype(np.float64)
    got = gl.backward_quant(f, dh, f["h"], f["v"], params, f["masks"].arr)["dh0"]
    assert np.linalg.norm(got - want) < 1.5e-7 * np.linalg.norm(want)
