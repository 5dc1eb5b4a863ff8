"""Small Rice shards, decoded a warp each when there are many of them: sizes
around the limit, bodies longer than the warp's staging, and every kind of bad
end, in lists long enough -- the GPU must accept what the oracle accepts."""

import numpy as np
import pytest
import torch

import oracle
from fastvid_b200 import synth
from fastvid_b200.batch import BatchCodec
from test_rice_parallel_gpu import PATTERNS, _stream

pytestmark = pytest.mark.gpu

MANY = 148 * 12 + 30  # small shards above which they no longer get a CTA each
SIZES = ((32, 32), (31, 33), (16, 16), (8, 16), (33, 3), (5, 1), (3, 1), (1, 1))


def _symbols(pattern, n, k, top, rng):
    mid = min(top, (1 << k) + (0x1555 & ((1 << k) - 1)))
    v = {"constant": np.full(n, mid), "two": np.where(np.arange(n) // 4 % 2, mid, mid ^ 1),
         "random": rng.integers(0, 3 << k, n), "zeros": np.zeros(n, dtype=np.int64),
         "spikes": np.where(rng.random(n) < 0.01, min(top, 300 << k), rng.integers(0, 2 << k, n))}[pattern]
    return np.minimum(v, top).astype(int).tolist()


def _device(stream):
    return torch.frombuffer(bytearray(stream), dtype=torch.uint8).cuda()


@pytest.mark.parametrize("depth", (12, 16))
def test_hand_made_lanes(cuda, depth):
    rng = np.random.default_rng(depth)
    top = 2 * ((1 << depth) - 1)
    good, bad = [], []
    for k in (0, 1, 3, 8, 12, 16):
        for pattern in PATTERNS:
            for width, height in SIZES:
                v = _symbols(pattern, width * height, k, top, rng)
                if sum(x >> k for x in v) > 300_000:  # a body's length is 16 bits
                    continue
                good.append(_stream(v, k, depth, width, height))
                if (width, height) in ((32, 32), (8, 16), (5, 1)):
                    bad += [_stream(v, k, depth, width, height, tail=[1] + [0] * k),
                            _stream(v, k, depth, width, height, tail=[0] * 9),
                            _stream(v, k, depth, width, height, cut=1)]
                    if pattern == "random":
                        v[-1 - int(rng.integers(0, min(8, len(v))))] = top + 1
                        bad.append(_stream(v, k, depth, width, height))
    good = [s for s in good if len(s) - 67 < 65536]
    expected = [oracle.decode(s) for s in good]
    codec = BatchCodec(cuda, use_graphs=False)
    many = [_device(s) for s in good] * (-(-MANY // len(good)))
    for i, planes in enumerate(codec.decode(many)):
        assert np.array_equal(planes[0].cpu().numpy(), expected[i % len(good)][0])
    rejected = 0
    for i in rng.permutation(len(bad))[:60]:
        try:
            want = oracle.decode(bad[i])
        except Exception:
            want = None
            rejected += 1
        streams = many[:5] + [_device(bad[i])] + many[5:]
        if want is None:
            with pytest.raises(RuntimeError, match="frame 5:"):
                codec.decode(streams)
        else:
            assert np.array_equal(codec.decode(streams)[5][0].cpu().numpy(), want[0])
    assert rejected > 20


@pytest.mark.parametrize("tile", ((32, 32), (16, 16), (25, 41), (64, 17)))
def test_frames_of_many_small_shards(cuda, tile):
    """1,025 and 1,088 symbols a tile are above the limit, their edge tiles below."""
    for layout, depth in (("gray", 8), ("yuv422", 8), ("gray", 16)):
        planes = synth.make_frame(2049, 1055, layout, depth, tile[0])
        kw = dict(layout=layout, bit_depth=depth, quality=100, tile_size=tile)
        codec = BatchCodec(cuda)
        stream = codec.encode([tuple(torch.from_numpy(p).to(cuda) for p in planes)], **kw)[0]
        assert bytes(stream.cpu().numpy()) == oracle.encode(planes, threads=oracle.cpu_threads(), **kw)
        for a, b in zip(codec.decode([stream])[0], planes):
            assert np.array_equal(a.cpu().numpy(), b)
