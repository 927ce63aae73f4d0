"""The recurrences with a thread per hidden unit (QuantLSTM up to 128 units, QuantGRU up to 256, 8 and 16 bits) and over clusters: the edges of widths, of rows per CTA
or cluster and of step counts, every form of what a forward saves, against the CPU checkers."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest
import torch

import gpu_lib as gl
import lstm_lib as ll
import oracle_lib as ol
from rx_met_b200 import _cabi, _cabi_lstm as L
from test_gru_gpu import (CONFIGS, calibrated, test_forward_quant_matches_restatement as gru_forward_matches,
                          test_packed_step_flags_equal_the_byte_masks as packed_flags_match)
from test_lstm_gpu import dev, mod, torch_args
from test_lstm_wide_gpu import setup, test_wide_forward_is_bit_exact as lstm_forward_matches

pytestmark = pytest.mark.gpu


# one, two and four rows of a CTA (128 units; twice that at 64), the last CTA partly empty; one byte plane and two
@pytest.mark.parametrize("abits", [8, 16])
@pytest.mark.parametrize("T,B,I,H", [(1, 1, 3, 1), (2, 149, 5, 65), (3, 148, 7, 128), (2, 593, 6, 127), (4, 3, 9, 33), (2, 1185, 4, 64), (3, 593, 5, 63)])
def test_lstm_units(T, B, I, H, abits):
    lstm_forward_matches(T, B, I, H, 8, abits, L.PER_CHANNEL, True, True)


# the same on one byte plane, which takes its calls from 24 (up to 32 units 128) steps on
@pytest.mark.parametrize("T,B,I,H", [(32, 149, 5, 65), (33, 148, 7, 128), (32, 297, 6, 100), (32, 593, 6, 127), (32, 1185, 4, 64), (33, 593, 5, 63), (128, 3, 4, 20)])
def test_lstm_units_on_one_plane(T, B, I, H):
    lstm_forward_matches(T, B, I, H, 8, 8, L.PER_CHANNEL, True, True)


@pytest.mark.parametrize("keep", [("gate_outputs", "cell_states_clamped"), ("weight_hh_linear_clamped", "hidden_outputs"), ("weight_ih_linear",)])
@pytest.mark.parametrize("abits", [8, 16])
def test_lstm_units_save_what_is_asked_for(abits, keep):
    T, B, I, H = 25, 5, 7, 100
    p, box, _ = setup(T, B, I, H, 8, abits, L.PER_CHANNEL, True, True)
    q = ll.quantize_masters("orc", p, box)
    _, _, _, want, want_mask = ll.forward_quantized_masked(box, T, B, q, exact_sums=True)
    a = {n: dev(p[n]) for n in ("w_ih", "w_hh", "b_ih", "b_hh", "x", "h0", "c0")}
    wide = ("weight_ih_linear", "weight_hh_linear", "gate_inputs", "gate_outputs")
    shape = lambda n: (T, B, 4 * H if n.replace("_clamped", "") in wide else H)  # noqa: E731
    got = {n: torch.full(shape(n), 77, dtype=torch.uint8 if n.endswith("_clamped") else torch.float32, device="cuda") for n in keep}
    trace = L.Trace(**{n: t.data_ptr() for n, t in got.items()})
    out, hn, cn = torch.empty(T, B, H, device="cuda"), torch.empty(B, H, device="cuda"), torch.empty(B, H, device="cuda")
    lib = mod()._library()
    work = torch.empty(lib.rxmet_lstm_workspace_bytes(1, T, B, I, H), dtype=torch.uint8, device="cuda")
    ptr = lambda t: C.c_void_p(t.data_ptr())  # noqa: E731
    rc = lib.rxmet_lstm_forward_quantized(T, B, I, H, *[ptr(a[n]) for n in ("w_ih", "w_hh", "b_ih", "b_hh", "x", "h0", "c0")], C.byref(box.struct), 0,
                                          ptr(out), ptr(hn), ptr(cn), C.byref(trace), None, ptr(work), C.c_size_t(work.numel()),
                                          C.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    for n, t in got.items():
        oracle = want_mask[n[:-8]] if n.endswith("_clamped") else want[n]
        np.testing.assert_array_equal(t.cpu().numpy(), oracle, err_msg=n)


# 32 units: 4, 8, 16 rows of a CTA; 64: 2, 4, 8; 128: 1, 2, 4; clusters beyond: 4, 8
@pytest.mark.parametrize("T,B,I,H", [(1, 1, 3, 1), (2, 1185, 4, 32), (2, 2369, 3, 31), (3, 593, 4, 33), (2, 1185, 5, 64), (4, 149, 6, 65), (3, 593, 4, 128),
                                     (2, 131, 5, 129), (3, 265, 4, 192), (2, 265, 7, 193), (5, 3, 5, 256), (2, 265, 4, 255)])
def test_gru_units(T, B, I, H):
    gru_forward_matches(gl, "a16", (T, B, I, H))


# one plane of signed codes: 64 units: 2, 4, 8 rows of a CTA; 128: 1, 2, 4; clusters beyond: 4, 8
@pytest.mark.parametrize("T,B,I,H", [(64, 100, 4, 33), (16, 700, 3, 50), (40, 101, 5, 64), (16, 1185, 3, 64), (64, 1, 6, 65), (16, 149, 6, 65), (16, 593, 4, 128),
                                     (17, 601, 3, 100), (2, 131, 5, 129), (2, 500, 4, 129), (2, 421, 5, 192), (3, 265, 7, 193), (5, 3, 5, 256), (2, 301, 4, 255)])
def test_8bit_gru_units(T, B, I, H):
    gru_forward_matches(gl, "w8a8", (T, B, I, H))


@pytest.mark.parametrize("shape", [(17, 9, 40, 128), (16, 601, 8, 64), (40, 130, 8, 64)], ids=lambda s: "x".join(map(str, s)))
def test_8bit_gru_units_pack_their_flags(monkeypatch, shape):
    packed_flags_match(monkeypatch, shape)


@pytest.mark.parametrize("cfg_name,T,B,I,H", [("a16", 3, 5, 6, 64), ("a16", 2, 150, 4, 100), ("a16", 3, 9, 5, 200), ("w8a8", 40, 130, 6, 64), ("w8a8", 64, 9, 4, 100),
                                              ("w8a8", 16, 300, 4, 60), ("w8a8", 3, 9, 5, 200)])
def test_gru_units_save_what_is_asked_for(cfg_name, T, B, I, H):
    from rx_met_b200 import gru_interface_binding as m
    prob, params = calibrated((T, B, I, H), seed=T + B + H, cfg=ol.make_config(**CONFIGS[cfg_name]), with_h0=True)
    want = ol.forward_quant("orc", *prob, params, training=True)
    p = m.GRUQuantParams._from_c(params.c, [params.chan["scale_" + n].tolist() for n in ("W", "R", "bw", "br")])
    for training in (False, True):
        out = [t.cpu().numpy() for t in m.forward_quant_int_storage(training, T, B, I, H, *[gl.dev(a) for a in prob], p)]
        assert np.array_equal(out[0], want["h"]) and np.array_equal(out[1], want["v"])
        for name, flags in zip(_cabi.MASK_NAMES, out[7:]):
            assert flags.size == 0 if not training else np.array_equal(flags, want["masks"].arr[name]), name


# clusters with one to three row groups that run on their own: every number of rows, groups and clusters partly empty
@pytest.mark.parametrize("T,B,H", [(3, 5, 512), (2, 67, 512), (2, 130, 512), (3, 201, 500), (2, 257, 512), (1, 390, 410), (2, 701, 512), (4, 9, 129), (2, 131, 256),
                                   (3, 261, 200), (2, 401, 256)])
def test_lstm_clusters(T, B, H):
    lstm_forward_matches(T, B, 6, H, 8, 16, L.PER_CHANNEL, True, True)
