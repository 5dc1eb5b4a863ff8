"""The wavefront kernels when warps and warp pairs take more than one tile of
several bands, against the oracle: equal bytes and equal planes."""

import numpy as np
import pytest
import torch

import fastvid_b200
import oracle
from fastvid_b200 import autotune, synth
from test_wavefront_gpu import FORMATS, _check

pytestmark = pytest.mark.gpu


def _tall_tiles(count, tile_w, layout, depth, seed, rows):
    """A frame of at least `count` tiles of tile_w x 65 samples (two bands) with
    edge tiles of other sizes."""
    planes = 1 if layout == "gray" else 3
    cols = -(-count // (planes * rows))
    return synth.make_frame(cols * tile_w - 3, rows * 65 - 7, layout, depth, seed)


@pytest.mark.parametrize("layout,depth,quality", FORMATS[:-1])
def test_warps_take_tiles_from_the_queue(cuda, layout, depth, quality):
    """Half as many tiles again as the GPU runs warps (four CTAs of four on an
    SM): windows and carry rows are used for a second tile, of odd and even width."""
    warps = 16 * torch.cuda.get_device_properties(cuda).multi_processor_count
    tile_w = 22 if depth == 10 else 19
    planes = _tall_tiles(warps * 3 // 2, tile_w, layout, depth, depth, 30)
    kw = dict(layout=layout, bit_depth=depth, quality=quality, tile_size=(tile_w, 65))
    expected = oracle.encode(planes, threads=oracle.cpu_threads(), **kw)
    got = fastvid_b200.encode(tuple(torch.from_numpy(p).to(cuda) for p in planes), **kw)
    assert bytes(got.cpu().numpy()) == expected
    for a, b in zip(fastvid_b200.decode(got), oracle.decode(expected, threads=oracle.cpu_threads())):
        assert np.array_equal(a.cpu().numpy(), b)


@pytest.mark.parametrize("layout,depth,quality", FORMATS[:-1])
def test_pairs_go_round(cuda, layout, depth, quality):
    """One CTA an SM and about 2.5 tiles an SM: a CTA's two pairs take a tile each
    and some a second one, of 1 to 4 bands."""
    sms = torch.cuda.get_device_properties(cuda).multi_processor_count
    tile_w = 40 if depth == 12 else 37
    planes = _tall_tiles(sms * 5 // 2, tile_w, layout, depth, 3 * depth, 10)
    try:
        autotune.set_launch({"enc_predict": 1, "dec_reconstruct": 1})
        for tile_h in (65, 200):
            count = oracle.geometry(planes[0].shape[1], planes[0].shape[0], {"gray": 0, "yuv422": 1, "rgb444": 2}[layout],
                                    (tile_w, tile_h))[0]
            if tile_h == 65:
                assert 2 * sms < count <= 3 * sms
            _check(planes, tuple(torch.from_numpy(p).to(cuda) for p in planes), layout=layout, bit_depth=depth,
                   quality=quality, tile_size=(tile_w, tile_h))
    finally:
        autotune.reset_launch()
