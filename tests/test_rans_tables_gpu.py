"""rANS shards over the sizes of their tables -- up to 36 symbols (entries in
shared memory), up to 170 (bucket table in the record), up to 255 (built by the
decoder), values of eight bits and wider, values above the encoder's local
table -- and over few shards (tables of all slots) and many: lossless frames
come back exactly, and small ones equal the oracle's streams byte for byte."""

import numpy as np
import pytest
import torch

import fastvid_b200
import oracle
from fastvid_b200 import autotune
from fastvid_b200.batch import BatchCodec

pytestmark = pytest.mark.gpu

# spread of the residuals, about a third of the distinct symbols
SPREADS = (0, 2, 10, 17, 40, 55, 80, 84)


def _planes(width, height, depth, spread, seed, device):
    """Planes whose prediction residuals lie within +-spread: random samples in
    a band of width spread (the gradient of such samples stays in the band)."""
    gen = torch.Generator(device="cpu")
    gen.manual_seed(seed)
    mid = 1 << (depth - 1)
    return tuple((torch.randint(0, spread + 1, (height, width), generator=gen) + mid).to(torch.int32).to(torch.uint16)
                 .to(device) for _ in range(3))


@pytest.mark.parametrize("spread", SPREADS)
def test_small_frames_match_the_oracle(cuda, spread):
    for depth in (8, 12, 16):
        planes = _planes(101, 83, depth, spread, 7 * spread + depth, cuda)
        kw = dict(layout="rgb444", bit_depth=depth, quality=100, tile_size=(64, 64))
        stream = fastvid_b200.encode(planes, **kw)
        assert bytes(stream.cpu().numpy()) == oracle.encode(tuple(p.cpu().numpy() for p in planes), **kw)
        for a, b in zip(fastvid_b200.decode(stream), planes):
            assert np.array_equal(a.cpu().numpy(), b.cpu().numpy())


@pytest.mark.parametrize("depth", (12, 16))
def test_many_shards_of_all_table_sizes(cuda, depth):
    """2,300 shards and more: whole warps of one table size, mixed warps, ragged shards."""
    frames = [_planes(901, 507, depth, s, 100 + s, cuda) for s in SPREADS]
    codec = BatchCodec(cuda)
    streams = codec.encode(frames, layout="rgb444", bit_depth=depth, quality=100, tile_size=(128, 96))
    for frame, planes in zip(frames, codec.decode(streams)):
        for a, b in zip(planes, frame):
            assert torch.equal(a.view(torch.int16), b.view(torch.int16))


def test_warps_that_take_several_groups(cuda):
    """One CTA an SM, about three groups of eight shards a warp: a table that
    the four lanes build takes the place of one that they copied, and back."""
    warps = 4 * torch.cuda.get_device_properties(cuda).multi_processor_count
    rows = -(-3 * 8 * warps // (3 * 22)) * 64  # 22 shards of 64x64 samples a row of tiles, three planes
    planes = []
    for p in range(3):
        gen = torch.Generator(device="cpu")
        gen.manual_seed(p)
        spread = torch.tensor([105, 2, 10, 80, 105, 17, 2, 55, 105]).repeat(1000)
        tiles = torch.rand(rows // 64, 64, 22, 64, generator=gen)
        tiles *= spread[:tiles.shape[0] * 22].view(-1, 1, 22, 1) + 1
        planes.append(tiles.to(torch.int32).view(rows, 22 * 64).to(torch.uint16).to(cuda))
    codec = BatchCodec(cuda)
    streams = codec.encode([planes], layout="rgb444", bit_depth=12, quality=100, tile_size=(64, 64))
    try:
        autotune.set_launch({"dec_rans": 1})
        decoded = codec.decode(streams)[0]
    finally:
        autotune.reset_launch()
    for a, b in zip(decoded, planes):
        assert torch.equal(a.view(torch.int16), b.view(torch.int16))


@pytest.mark.parametrize("depth", (12, 16))
def test_neighbouring_shards_of_different_tables(cuda, depth):
    """The eight shards of an encoder warp with a table of their own each,
    within the local table and above it, some of them ragged."""
    gen = torch.Generator(device="cpu")
    gen.manual_seed(depth)
    spread = torch.tensor([105, 2, 40, 10, 80, 0, 17, 55, 84]).repeat(8)[:64]
    planes = []
    for p in range(3):
        tiles = torch.rand(8, 64, 8, 64, generator=gen) * (spread.roll(p).view(8, 1, 8, 1) + 1)
        planes.append(tiles.to(torch.int32).view(512, 512)[:509, :507].numpy().astype(np.uint16))
    kw = dict(layout="rgb444", bit_depth=depth, quality=100, tile_size=(64, 64))
    stream = fastvid_b200.encode(tuple(torch.from_numpy(p.copy()).to(cuda) for p in planes), **kw)
    assert bytes(stream.cpu().numpy()) == oracle.encode(tuple(np.ascontiguousarray(p) for p in planes), **kw)
    for a, b in zip(fastvid_b200.decode(stream), planes):
        assert np.array_equal(a.cpu().numpy(), b)


def test_short_shards_of_all_table_sizes(cuda):
    """More shards than dec_rans gives room for whole tables: tables within the
    small local room, above it, and built by the decoder, narrow and wide."""
    gen = torch.Generator(device="cpu")
    gen.manual_seed(4)
    rows, cols = 133, 72  # tiles of 32x16, three planes: 28,728 shards
    spread = torch.tensor([120, 2, 10, 80, 115, 17, 0, 40, 120, 30, 7])
    planes = []
    for p in range(3):
        tiles = torch.rand(rows, 16, cols, 32, generator=gen)
        tiles *= spread[(torch.arange(rows * cols) + p) % len(spread)].view(rows, 1, cols, 1) + 1
        planes.append(tiles.to(torch.int32).view(rows * 16, cols * 32).to(torch.uint16).to(cuda))
    codec = BatchCodec(cuda)
    streams = codec.encode([planes], layout="rgb444", bit_depth=12, quality=100, tile_size=(32, 16))
    for a, b in zip(codec.decode(streams)[0], planes):
        assert torch.equal(a.view(torch.int16), b.view(torch.int16))
    # and as the only frames of their kind (tables of all slots), in the oracle's bytes
    part = tuple(p[:64, :160].contiguous() for p in planes)
    kw = dict(layout="rgb444", bit_depth=12, quality=100, tile_size=(32, 16))
    stream = fastvid_b200.encode(part, **kw)
    assert bytes(stream.cpu().numpy()) == oracle.encode(tuple(p.cpu().numpy() for p in part), **kw)
    for a, b in zip(fastvid_b200.decode(stream), part):
        assert torch.equal(a.view(torch.int16), b.view(torch.int16))


@pytest.mark.parametrize("tiles", ((24, 28), (5, 9)))
def test_tables_around_the_bucket_limit(cuda, tiles):
    """Tables of some 160 to 185 symbols, in many shards and in few: with more
    than 170 the decoder builds the bucket table itself."""
    gen = torch.Generator(device="cpu")
    gen.manual_seed(11)
    rows, cols = tiles
    spread = torch.arange(81, 95).repeat(rows * cols)
    planes = []
    for p in range(3):
        t = torch.rand(rows, 64, cols, 64, generator=gen) * (spread[p:p + rows * cols].view(rows, 1, cols, 1) + 1)
        planes.append(t.to(torch.int32).view(rows * 64, cols * 64).to(torch.uint16).to(cuda))
    kw = dict(layout="rgb444", bit_depth=12, quality=100, tile_size=(64, 64))
    codec = BatchCodec(cuda)
    stream = codec.encode([planes], **kw)[0]
    for a, b in zip(codec.decode([stream])[0], planes):
        assert torch.equal(a.view(torch.int16), b.view(torch.int16))
    # the streams do hold tables on both sides of the limit
    data = stream.cpu().numpy()
    counts = set()
    for t in range(int.from_bytes(data[28:32].tobytes(), "little")):
        off = int.from_bytes(data[52 + 32 * t:60 + 32 * t].tobytes(), "little")
        if data[off] == 19:
            counts.add((int(data[off + 4]) & 127) + (int(data[off + 5]) << 7 if data[off + 4] & 128 else 0))
    assert any(c <= 170 for c in counts) and any(170 < c <= 176 for c in counts) and any(c > 176 for c in counts)
