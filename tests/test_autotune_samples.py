"""The samples that the autotuner times its knobs on (host code only)."""

import ctypes

from fastvid_b200 import _native, autotune, synth


def test_wide_symbol_sample_makes_a_u32_batch():
    """The wavefront block and the warps per tile act on u32 batches alone, so
    their sample must be one; the mix itself is not."""
    lib = _native.load()
    specs = synth.mixed_batch_specs(12)
    idx, params = autotune.wide_symbol_sample(specs)
    assert idx and params["quality"] == 100

    def fold16(frames):
        bucket = _native.Bucket()
        _native.check(lib.fvb_batch_bucket((_native.Frame * len(frames))(*frames), len(frames), ctypes.byref(bucket)))
        return bucket.fold16

    def plan(spec, quality):
        frame = _native.Frame()
        layout = {"gray": 0, "yuv422": 1, "rgb444": 2}[spec["layout"]]
        _native.check(lib.fvb_encode_plan(spec["width"], spec["height"], layout, spec["bit_depth"], quality, 24, 1, 64,
                                          64, ctypes.byref(frame), None))
        return frame

    assert fold16([plan(s, s["quality"]) for s in specs]) == 1
    assert fold16([plan(specs[i], params["quality"]) for i in idx]) == 0
