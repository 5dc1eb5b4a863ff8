"""Lists whose planes must be copied to be read row by row: the copies live
until the encoder has read them."""

import pytest
import torch

import oracle
from fastvid_b200 import synth
from fastvid_b200.batch import BatchCodec

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graphs", (False, True))
@pytest.mark.parametrize("layout,depth,quality", (("gray", 8, 100), ("rgb444", 10, 90)))
def test_transposed_and_strided_planes(cuda, graphs, layout, depth, quality):
    kw = dict(layout=layout, bit_depth=depth, quality=quality, tile_size=(64, 64))
    frames, expected = [], []
    for seed in range(6):
        planes = synth.make_frame(190, 133, layout, depth, seed)
        expected.append(oracle.encode(planes, **kw))
        views = []
        for p in planes:
            t = torch.from_numpy(p.astype("int32")).to(cuda)
            if seed % 2:
                view = t.t().contiguous().to(torch.uint16).t()                      # column by column
            else:
                view = torch.stack((t, t * 0), dim=2).to(torch.uint16)[:, :, 0]     # every other sample
            assert view.stride(1) != 1
            views.append(view)
        frames.append(tuple(views))
    codec = BatchCodec(cuda, use_graphs=graphs)
    for _ in range(2):
        for stream, want in zip(codec.encode(frames, **kw), expected):
            assert bytes(stream.cpu().numpy()) == want
