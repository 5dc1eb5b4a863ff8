"""Tile placement as the kernels compute it (host code only): offsets are the
running sums over the tiles, whatever the size of a tile."""

import ctypes

import pytest

from fastvid_b200 import _native


def _tiles(w, h, layout, tile):
    lib = _native.load()
    frame = _native.Frame()
    _native.check(lib.fvb_encode_plan(w, h, layout, 8, 90, 24, 1, *tile, ctypes.byref(frame), None))
    for t in range(frame.tiles):
        g = (ctypes.c_int64 * 8)()
        _native.check(lib.fvb_tile_geometry(ctypes.byref(frame), t, g))
        yield list(g)
    assert lib.fvb_tile_geometry(ctypes.byref(frame), frame.tiles, (ctypes.c_int64 * 8)()) != 0
    assert lib.fvb_tile_geometry(ctypes.byref(frame), -1, (ctypes.c_int64 * 8)()) != 0


@pytest.mark.parametrize("w,h,layout,tile", [
    (300, 200, 0, (64, 64)),
    (301, 203, 1, (67, 35)),
    (263, 133, 2, (32, 128)),
    (1300, 90, 1, (600, 40)),
    (65536, 32769, 0, (65535, 32769)),    # tiles of more than 2^31 samples
    (131071, 65535, 1, (65535, 65535)),   # more than 2^32 - 2^17, subsampled planes
    (140000, 131071, 2, (65535, 65535)),  # several of them, in two rows
])
def test_offsets_are_the_sums_over_the_tiles(w, h, layout, tile):
    samples = shards = 0
    x = y = plane = 0
    for i, (p, gx, gy, gw, gh, first_sample, first_shard, count) in enumerate(_tiles(w, h, layout, tile)):
        pw = (w + 1) // 2 if layout == 1 and p else w
        tw = (tile[0] + 1) // 2 if layout == 1 and p else tile[0]
        if p != plane:
            assert p == plane + 1
            plane, x, y = p, 0, 0
        assert (gx, gy) == (x, y)
        assert (gw, gh) == (min(tw, pw - x), min(tile[1], h - y))
        assert (first_sample, first_shard) == (samples, shards), i
        assert count == -(-gw * gh // 4096)
        samples += -(-gw * gh // 8) * 8
        shards += count
        x += tw
        if x >= pw:
            x, y = 0, y + tile[1]
    assert plane == (2 if layout else 0) and y >= h and x == 0
