"""The tensor-core input projection on byte planes at the edges of its tiles: slices of weight tiles (256 k-bytes), row tiles of 128 and 64, shares
of the channel tiles of few row tiles, and several row tiles of a CTA, against the CPU checkers (codes, hence exact)."""
from __future__ import annotations

import pytest

import gpu_lib as gl
from rx_met_b200 import _cabi_lstm as L
from test_gru_gpu import test_forward_quant_matches_restatement as gru_forward_matches
from test_lstm_wide_gpu import test_wide_forward_is_bit_exact as lstm_forward_matches

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,B,I,H", [(1, 1, 1, 43), (2, 63, 255, 40), (3, 43, 256, 43), (1, 64, 257, 86), (2, 97, 288, 20), (1, 129, 511, 22), (3, 70, 512, 43),
                                     (3, 16900, 5, 5), (2, 9500, 300, 6)])
def test_gru_projection(T, B, I, H):
    gru_forward_matches(gl, "a16", (T, B, I, H))


@pytest.mark.parametrize("abits", [8, 16])
@pytest.mark.parametrize("T,B,I,H", [(1, 1, 1, 32), (2, 64, 256, 33), (1, 129, 255, 512), (3, 13000, 4, 3)])
def test_lstm_projection(T, B, I, H, abits):
    lstm_forward_matches(T, B, I, H, 4, abits, L.PER_CHANNEL, True, True)


# 8-bit codes (input_proj_umma.cu): many rows on channel counts that leave the last tile partly empty
@pytest.mark.parametrize("T,B,I,H", [(21, 400, 13, 37), (12, 700, 40, 20), (9, 1000, 5, 85), (3, 2800, 64, 100)])
def test_8bit_gru_projection_of_partly_empty_tiles(T, B, I, H):
    gru_forward_matches(gl, "w8a8", (T, B, I, H))
