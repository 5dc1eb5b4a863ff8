"""The wavefront kernels at the sizes where they can go wrong -- tile widths
around the 8-sample chunks, the 32-column blocks and the widest tile, heights
around the 64-row bands, plane views whose rows start at every alignment, few
and many tiles -- against the oracle: equal bytes and equal planes."""

import numpy as np
import pytest
import torch

import fastvid_b200
import oracle
from fastvid_b200 import synth

pytestmark = pytest.mark.gpu

WIDTHS = (1, 2, 7, 8, 9, 31, 32, 33, 35, 62, 64, 65, 96, 127, 128, 130, 255, 256, 257, 511, 512)
HEIGHTS = (1, 2, 63, 64, 65, 129, 250)
FORMATS = (("gray", 8, 100), ("gray", 10, 90), ("gray", 12, 30), ("gray", 16, 87), ("yuv422", 10, 90),
           ("rgb444", 8, 66), ("rgb444", 12, 1), ("rgb444", 16, 50), ("gray", 16, 100))


def _check(planes, cuda_planes, **kw):
    expected = oracle.encode(planes, **kw)
    got = fastvid_b200.encode(cuda_planes, **kw)
    assert bytes(got.cpu().numpy()) == expected, kw
    for a, b in zip(fastvid_b200.decode(got), oracle.decode(expected)):
        assert np.array_equal(a.cpu().numpy(), b), kw


def _view(plane, cuda, lead, gap):
    """The plane as a view of a larger tensor: rows start `lead` samples after
    a 16-byte boundary (the first one) and `gap` samples apart."""
    h, w = plane.shape
    big = torch.full((h * (w + gap) + lead + 8,), 0xFFFF, dtype=torch.int32).to(torch.uint16).to(cuda)
    view = big[lead:lead + h * (w + gap)].view(h, w + gap)[:, :w]
    view.copy_(torch.from_numpy(plane).to(cuda))
    return view


@pytest.mark.parametrize("width", WIDTHS)
def test_tile_widths_and_heights(cuda, width):
    for i, height in enumerate(HEIGHTS):
        layout, depth, q = FORMATS[(WIDTHS.index(width) + i) % len(FORMATS)]
        planes = synth.make_frame(width, height, layout, depth, 100 * width + height)
        _check(planes, tuple(torch.from_numpy(p).to(cuda) for p in planes), layout=layout, bit_depth=depth, quality=q,
               tile_size=(512, 256))


@pytest.mark.parametrize("layout,depth,quality", FORMATS)
def test_row_alignments(cuda, layout, depth, quality):
    for lead, gap, width in ((0, 8, 130), (1, 0, 131), (2, 6, 128), (3, 5, 129), (5, 1, 67), (6, 2, 66), (7, 9, 72)):
        planes = synth.make_frame(width, 70, layout, depth, 7 * lead + gap)
        _check(planes, tuple(_view(p, cuda, lead, gap) for p in planes), layout=layout, bit_depth=depth,
               quality=quality, tile_size=(64, 128))


@pytest.mark.parametrize("layout,depth,quality", FORMATS)
def test_many_tiles(cuda, layout, depth, quality):
    """More tiles than the GPU has warps for."""
    planes = synth.make_frame(1251, 1203, layout, depth, 11)
    _check(planes, tuple(torch.from_numpy(p).to(cuda) for p in planes), layout=layout, bit_depth=depth,
           quality=quality, tile_size=(34, 33) if layout == "gray" else (48, 66))


@pytest.mark.parametrize("depth,quality", ((8, 66), (10, 1), (12, 1), (12, 50), (16, 99)))
def test_extreme_samples_saturate_alike(cuda, depth, quality):
    """Alternating extremes: the largest residuals of either sign."""
    rng = np.random.default_rng(depth)
    maximum = (1 << depth) - 1
    planes = tuple((rng.integers(0, 2, (97, 145)) * maximum).astype(np.uint16) for _ in range(3))
    _check(planes, tuple(torch.from_numpy(p).to(cuda) for p in planes), layout="rgb444", bit_depth=depth,
           quality=quality, tile_size=(128, 64))
