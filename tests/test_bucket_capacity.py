"""Capacities in the terms of the frames' own counts, and plans of frames that
were never planned (host code only)."""

import ctypes
import subprocess
import sys

import pytest

from fastvid_b200 import _native
from fastvid_b200._native import Bucket, Frame


def _frame(width, height, layout, depth, quality, tile):
    frame = Frame()
    _native.check(_native.load().fvb_encode_plan(width, height, layout, depth, quality, 24, 1, *tile,
                                                 ctypes.byref(frame), None))
    return frame


@pytest.mark.parametrize("args", [(67, 35, 0, 8, 100, (256, 128)), (263, 133, 1, 10, 90, (33, 17)),
                                  (101, 83, 2, 12, 90, (1, 3)), (1300, 90, 0, 16, 90, (600, 40))])
def test_a_bucket_of_the_frames_own_sums_takes_them(args):
    """Tiles are padded in the workspace; a capacity still counts samples."""
    lib = _native.load()
    frames = (Frame * 3)(*[_frame(*args)] * 3)
    f = frames[0]
    rounded = Bucket()
    _native.check(lib.fvb_batch_bucket(frames, 3, ctypes.byref(rounded)))
    own = Bucket()
    ctypes.memmove(ctypes.byref(own), ctypes.byref(rounded), ctypes.sizeof(own))  # passes and flags
    own.frames, own.tiles, own.shards = 3, 3 * f.tiles, 3 * f.shards
    own.samples, own.prefix = 3 * f.samples, 3 * f.prefix_bytes
    for p in range(own.passes):
        own.frames_p[p], own.tiles_p[p], own.shards_p[p] = 3, 3 * f.tiles, 3 * f.shards
        own.samples_p[p], own.prefix_p[p] = 3 * f.samples, 3 * f.prefix_bytes
    for plan, batch in ((lib.fvb_bucket_encode_plan, lib.fvb_batch_encode_plan),
                        (lib.fvb_bucket_decode_plan, lib.fvb_batch_decode_plan)):
        sizes = ctypes.c_int64(), ctypes.c_int64()
        _native.check(plan(ctypes.byref(own), ctypes.byref(sizes[0])))
        _native.check(batch(frames, 3, ctypes.byref(sizes[1])))
        assert sizes[0].value == sizes[1].value
    nulls = (ctypes.c_void_p * 9)()
    pitches = (ctypes.c_int64 * 9)()
    # it fits: the next check, of the workspace, is the one that fails
    assert lib.fvb_bucket_encode_prepare(ctypes.byref(own), frames, 3, nulls, pitches, None, 0, None) != 0
    assert _native.last_error() == "workspace is smaller than planned"
    own.samples -= 1
    assert lib.fvb_bucket_encode_prepare(ctypes.byref(own), frames, 3, nulls, pitches, None, 0, None) != 0
    assert _native.last_error() == "batch does not fit the bucket"


def test_an_unplanned_frame_does_not_end_the_process():
    code = """
import ctypes
from fastvid_b200 import _native
lib, frames, ws, bucket = _native.load(), (_native.Frame * 2)(), ctypes.c_int64(), _native.Bucket()
for plan in (lib.fvb_batch_encode_plan, lib.fvb_batch_decode_plan):
    assert plan(frames, 2, ctypes.byref(ws)) == 0 and ws.value > 0
assert lib.fvb_batch_bucket(frames, 2, ctypes.byref(bucket)) == 0
"""
    assert subprocess.run([sys.executable, "-c", code]).returncode == 0
