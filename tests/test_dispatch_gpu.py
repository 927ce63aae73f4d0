"""Which kernels calls of one operator take: the recurrences by steps, rows, width and what is saved, and the rows of a CTA beside large tables."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import lstm_lib as ll
from launch_lib import launches
from rx_met_b200 import _cabi, _cabi_lstm as L
from rx_met_b200 import gru_interface_binding as gru
from test_lstm_gpu import mod, torch_args

pytestmark = pytest.mark.gpu


def gru_call(T, B, I, H, training, bits=8):
    gen = torch.Generator().manual_seed(T + B + H)
    rand = lambda *shape: (torch.rand(shape, generator=gen) - 0.5).cuda()  # noqa: E731
    W, R, bw, br, x = rand(I, 3 * H), rand(H, 3 * H) * 0.2, rand(3 * H), rand(3 * H), rand(T, B, I)
    ranges = gru.GRUQuantizationRanges(H)
    gru.forward_calibrate(True, T, B, I, H, W, R, bw, br, x, None, "minmax", None, ranges)
    cfg = gru.OperatorQuantConfig()
    for name in _cabi.OP_NAMES:
        if name not in ("W", "R", "bw", "br"):
            setattr(cfg, f"{name}_", bits)
            setattr(cfg, f"{name}_symmetric_", False)
    params = gru.calculate_gru_quantitative_parameters(ranges, cfg)
    return lambda: gru.forward_quant_int_storage(training, T, B, I, H, W, R, bw, br, x, None, params)


def lstm_call(T, B, I, H, training, abits=8, wscale=1.0, times=1):
    """`times`: the batch repeated, beside parameters of one of it."""
    cfg = L.mixed_config(8, abits)
    p = ll.problem(T, B, I, H, seed=1, wscale=float(wscale / np.sqrt(H)))
    _, box = ll.calibrate("orc", cfg, p, np.stack([p["x"] * 0.8]))
    p.update(x=np.tile(p["x"], (1, times, 1)), h0=np.tile(p["h0"], (times, 1)), c0=np.tile(p["c0"], (times, 1)))
    m, args = mod(), torch_args(p)
    bundle = m._params_to_bundle(box)
    return lambda: m.lstm_forward_quantized(*args, False, bundle, "pedantic", False, training)


def launched(call, *names):
    """Of the kernels with one of these names in theirs: (name, CTAs, shared memory)."""
    return [(n, ctas, smem) for name, ctas, smem in launches(call) for n in names if n in name]


LANES, UNITS, BYTES = "recurrentLanesI8", "unitRecurrence", "recurrentQ"


# few steps or few rows: lanes, whose kernel has less to prepare
@pytest.mark.parametrize("T,B,H,training,expected", [
    (1, 1, 128, False, LANES), (4, 32, 80, False, LANES), (40, 1, 65, False, LANES), (64, 1, 65, False, UNITS), (20, 128, 128, False, LANES),
    (40, 128, 128, False, UNITS), (20, 200, 70, False, UNITS), (4, 300, 60, False, LANES), (20, 300, 60, False, UNITS), (98, 32, 64, False, LANES),
    (4, 64, 128, True, LANES), (16, 8, 70, True, UNITS), (4, 128, 64, True, LANES), (40, 128, 64, True, UNITS), (40, 900, 16, True, LANES)])
def test_8bit_gru_recurrence(T, B, H, training, expected):
    assert [n for n, _, _ in launched(gru_call(T, B, 8, H, training), LANES, UNITS)] == [expected]


@pytest.mark.parametrize("chunks,cell", [(None, "GruByteCell"), ("15,35,50", "GruUnitCell")])
def test_8bit_gru_beyond_128_units_in_time_chunks(monkeypatch, chunks, cell):
    """Asked for in time chunks, which the recurrence on bytes does not know: over clusters on byte planes, not in registers that spill."""
    call = gru_call(20, 16, 16, 192, False)
    if chunks:
        monkeypatch.setenv("RXMET_GRU_FWD_CHUNKS", chunks)
    assert [n for n, _, _ in launched(call, "GruByteCell", "GruUnitCell", "recurrentForwardI8")] == [cell]


# partly empty channel tiles: the tensor cores with many rows that fill them or have many inputs
@pytest.mark.parametrize("T,B,I,H,expected", [(98, 80, 40, 64, "inputLinearI8"), (98, 128, 40, 64, "inputProjUmma"), (98, 128, 8, 16, "inputLinearI8"),
                                              (98, 128, 8, 48, "inputLinearI8"), (98, 128, 40, 16, "inputProjUmma"), (2, 3, 8, 128, "inputProjUmma")])
def test_8bit_gru_projection(T, B, I, H, expected):
    assert [n for n, _, _ in launched(gru_call(T, B, I, H, False), "inputLinearI8", "inputProjUmma")] == [expected]


@pytest.mark.parametrize("T,B,H,training,expected", [
    (1, 1, 128, False, BYTES), (40, 1, 128, False, UNITS), (40, 16, 32, False, BYTES), (64, 16, 32, False, UNITS), (50, 1600, 12, False, BYTES),
    (8, 16, 100, True, BYTES), (40, 16, 100, True, UNITS), (64, 16, 32, True, BYTES), (130, 16, 32, True, UNITS), (40, 900, 40, True, BYTES)])
def test_8bit_lstm_recurrence(T, B, H, training, expected):
    assert [n for n, _, _ in launched(lstm_call(T, B, 5, H, training), BYTES, UNITS)] == [expected]


@pytest.mark.parametrize("wscale,ctas", [(1.0, 200), (8.0, 100)])
def test_rows_of_a_cta_beside_large_activation_tables(wscale, ctas):
    """Steep activations need 32 inputs a line: 120 kB of tables leave room for one CTA on an SM, and 400 rows run at the same time only with four a
    CTA instead of two."""
    (_, got, smem), = launched(lstm_call(2, 8, 5, 64, False, 16, wscale, times=50), UNITS)
    assert got == ctas and (smem > 114 * 1024) == (wscale > 1)
