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


def tile_shape(dims, f64, width, fine, side, points):
    f = _native.library().b200nufft_internal_tile_shape
    f.restype = ctypes.c_int
    out = (ctypes.c_int64 * 9)()
    axes = ctypes.c_int64 * 3
    f(dims, f64, width, axes(*fine), axes(*side), ctypes.c_int64(points), out)
    names = ("regs64", "tile0", "tile1", "tile2", "tiles", "padded_cells", "rows", "parts", "cap_parts")
    return dict(zip(names, out))


def shared_memory_tiles(width, fine, points):
    """Scratch bytes of cubic tiles of at most 100 KB, which are whole bins: a part
    of each tile and one per 2048 points, 592 at least."""
    tile = [min(16, 1 << (n - 1).bit_length()) for n in fine]
    padded = lambda: 16 * (tile[0] + width - 1) * (tile[1] + width - 1) * (tile[2] + width - 1)
    while padded() > 100 * 1024:
        tile[max(range(3), key=lambda a: (tile[a], a))] //= 2
    count = 1
    for a in range(3):
        count *= -(-fine[a] // tile[a])
    return (count + max(592, -(-points // 2048)) + 1) * padded()


@pytest.mark.parametrize("width", range(5, 14))
def test_3d_f64_register_tiles_reserve_no_more_than_shared_memory_tiles(width):
    """Register tiles are no whole number of bins, whose records therefore count
    in up to eight tiles; the scratch is bounded by the points all the same."""
    chosen = set()
    for fine in ((60, 50, 40), (128, 128, 128), (200, 180, 144), (400, 400, 400), (512, 512, 512)):
        for points in (2_000, 20_000, 150_000, 10**6, 10**7, 5 * 10**7, 2 * 10**8, 10**9):
            for side in ((2, 1, 1), (2, 2, 2), (2, 2, 4), (4, 4, 4), (4, 8, 8)):
                s = tile_shape(3, 1, width, fine, side, points)
                chosen.add(s["regs64"])
                assert s["rows"] <= 256
                if s["regs64"]:
                    held = s["parts"] * s["padded_cells"] * 16
                    assert held <= 1.1 * shared_memory_tiles(width, fine, points) + 128 * 2**20
                    # Parts of at least records / cap_parts records each, but for a tile's last.
                    assert s["parts"] <= s["tiles"] + s["cap_parts"] + 1
    assert chosen == {0, 1}, "sparse sets take the other tiles"
