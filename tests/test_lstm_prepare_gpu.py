"""Codes that a quantized LSTM call makes of its inputs, bit for bit: quotients at and next to a tie, outside the grid, beyond the range
of the short form, not finite; rows and columns that no vector divides; the checker divides in double."""
from __future__ import annotations

import numpy as np
import pytest

import lstm_lib as ll
from rx_met_b200 import _cabi_lstm as L
from test_lstm_gpu import mod, torch_args

pytestmark = pytest.mark.gpu


def awkward(shape, scale, zp, lo, hi, seed):
    """Ties of the whole grid and beyond it, their neighbours to both sides, values of every magnitude."""
    rng = np.random.default_rng(seed)
    n = int(np.prod(shape))
    k = rng.integers(lo - zp - 3, hi - zp + 4, n)
    v = ((k + 0.5) * np.float64(scale)).astype(np.float32)
    side = rng.integers(-2, 3, n)
    for _ in range(2):
        v = np.where(side > 0, np.nextafter(v, np.float32(np.inf)), np.where(side < 0, np.nextafter(v, np.float32(-np.inf)), v))
        side = side - np.sign(side)
    some = rng.random(n)
    v = np.where(some < 0.1, k * np.float64(scale), v).astype(np.float32)
    v = np.where((some >= 0.1) & (some < 0.2), np.float32(10.0) ** rng.uniform(-44, 38, n) * rng.choice([-1, 1], n), v).astype(np.float32)
    v[: min(n, 4)] = [0.0, -0.0, np.inf, -np.inf][: min(n, 4)]
    return v.reshape(shape)


@pytest.mark.parametrize("T,B,I,H,bits", [(3, 5, 40, 128, 16), (2, 3, 29, 33, 16), (1, 1, 1, 1, 16), (40, 2, 7, 32, 8), (2, 700, 256, 130, 12),
                                           (2, 9, 4, 512, 16), (48, 33, 128, 128, 8)])
def test_codes_of_the_inputs(T, B, I, H, bits):
    cfg = L.mixed_config(8, bits)
    p = ll.problem(T, B, I, H, seed=T + I, wscale=float(0.5 / np.sqrt(H)))
    _, box = ll.calibrate("orc", cfg, p, np.stack([p["x"]]))
    s, half = box.struct, 2 ** (bits - 1)
    for key, op in (("x", L.INPUT), ("h0", L.OUTPUT), ("c0", L.CELL_STATE)):
        p[key] = awkward(p[key].shape, s.scale[op], s.zero_point[op], -half, half - 1, seed=op)
    for key, scales in (("w_ih", box.channel_scales[0]), ("w_hh", box.channel_scales[1])):
        p[key] = (awkward(p[key].shape, 1.0, 0, -128, 127, seed=7) * np.asarray(scales, np.float32)[:, None]).astype(np.float32)
    want, clamped = ll.quantize_masters("orc", p, box, with_masks=True)
    got = mod().lstm_forward_quantized(*torch_args(p), False, mod()._params_to_bundle(box), "pedantic", False, True)[3]
    for name, key in (("input", "x"), ("h_0", "h0"), ("c_0", "c0"), ("weight_ih", "w_ih"), ("weight_hh", "w_hh"), ("bias_ih", "b_ih")):
        np.testing.assert_array_equal(got["quantized_master"][name].cpu().numpy().reshape(want[key].shape), want[key], err_msg=name)
        np.testing.assert_array_equal(got["master_clamp_masks"][name].cpu().numpy().reshape(want[key].shape).astype(np.uint8), clamped[key], err_msg=name)
