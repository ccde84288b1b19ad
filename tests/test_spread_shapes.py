"""Sizes that the spreader derives on the host, over everything a tuning
override accepts. No GPU."""

from __future__ import annotations

import ctypes

import pytest

from wgpunufft_b200 import _native


@pytest.mark.parametrize("width", range(5, 17))
def test_2d_f64_strip_counters_fit_their_tile(width):
    """The strips' record counters lie where the tile of sums goes afterwards:
    8 words per (strip, x start) and for the skipped records, strips of 16 x S
    starts whose windows reach 16 rows (24 from width 14)."""
    tile_bytes = _native.library().b200nufft_internal_strip64_tile_bytes
    tile_bytes.restype, tile_bytes.argtypes = ctypes.c_int64, [ctypes.c_int32] * 3
    rows = (16 if width <= 13 else 24) - width + 1
    sides = [1 << k for k in range(9)]
    for x in sides:
        for y in sides:
            counters = 4 * 8 * (-(-x // 16) * -(-y // rows) * 16 + 1)
            cells = 16 * (x + width - 1) * (y + width - 1)
            held = tile_bytes(width, x, y)
            assert held >= max(counters, cells), (width, x, y)
            assert held % 16 == 0
