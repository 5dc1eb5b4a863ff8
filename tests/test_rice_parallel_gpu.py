"""Rice shards built by hand, decoded by 32 threads a lane: periodic lanes in
which a wrong guess never falls in step (every part is then read again), long
quotients that span several parts, empty parts, and every kind of bad end.
The GPU must accept what the oracle accepts, with its planes."""

import numpy as np
import pytest
import torch

import fastvid_b200
import oracle

pytestmark = pytest.mark.gpu


def _lane(values, k, bits_more=()):
    bits = []
    for v in values:
        bits += [0] * (v >> k) + [1] + [(v >> i) & 1 for i in range(k)]
    bits += list(bits_more)
    bits += [0] * (-len(bits) % 8)
    return np.packbits(np.array(bits, dtype=np.uint8), bitorder="little").tobytes()


def _stream(symbols, k, depth, width, height, tail=(), cut=0):
    """A one-tile gray stream of one shard coded by Rice(k)."""
    n = width * height
    base = oracle.encode((np.zeros((height, width), dtype=np.uint16),), layout="gray", bit_depth=depth, quality=100,
                         tile_size=(width, height))
    lanes = [_lane(symbols[l::4], k, tail if l == 3 else ()) for l in range(min(4, n))]
    body = b"".join(len(x).to_bytes(4, "little") for x in lanes[:-1]) + b"".join(lanes)
    body = body[:len(body) - cut]
    record = bytes([1 + k]) + len(body).to_bytes(2, "little") + body
    head = bytearray(base[:64])
    head[60:64] = len(record).to_bytes(4, "little")
    return bytes(head) + record


def _check(stream):
    try:
        expected = oracle.decode(stream)
    except Exception:
        expected = None
    dev = torch.frombuffer(bytearray(stream), dtype=torch.uint8).cuda()
    if expected is None:
        with pytest.raises(RuntimeError):
            fastvid_b200.decode(dev)
        return False
    for a, b in zip(fastvid_b200.decode(dev), expected):
        assert np.array_equal(a.cpu().numpy(), b)
    return True


PATTERNS = ("constant", "two", "random", "spikes", "zeros")


@pytest.mark.parametrize("k", (0, 1, 3, 8, 12))
@pytest.mark.parametrize("pattern", PATTERNS)
def test_rice_lanes(cuda, k, pattern):
    rng = np.random.default_rng(17 * k + PATTERNS.index(pattern))
    accepted = 0
    for depth in (12, 16):
        top = 2 * ((1 << depth) - 1)
        for width, height in ((64, 64), (61, 67), (33, 3), (5, 1), (3, 1), (1, 1)):
            n = width * height
            if n > 4096:
                height, n = 4096 // width, width * (4096 // width)
            mid = min(top, (1 << k) + ((0x5555 >> 2) & ((1 << k) - 1)))
            v = {"constant": np.full(n, mid), "two": np.where(np.arange(n) // 4 % 2, mid, mid ^ 1),
                 "random": rng.integers(0, 3 << k, n), "zeros": np.zeros(n, dtype=np.int64),
                 "spikes": np.where(rng.random(n) < 0.003, min(top, 700 << k), rng.integers(0, 2 << k, n))}[pattern]
            v = np.minimum(v, top).astype(int).tolist()
            stream = _stream(v, k, depth, width, height)
            if len(stream) - 64 - 3 > 65535:
                continue
            accepted += _check(stream)
            # a code more, set padding, a missing byte
            for bad in (_stream(v, k, depth, width, height, tail=[1] + [0] * k),
                        _stream(v, k, depth, width, height, tail=[0] * 9),
                        _stream(v, k, depth, width, height, cut=1)):
                _check(bad)
    assert accepted >= 6


@pytest.mark.parametrize("k", (4, 8, 12))
def test_values_above_the_range_are_rejected(cuda, k):
    """One value at or just above the largest, near a lane's end: before the
    padding of its last byte and elsewhere."""
    rng = np.random.default_rng(k)
    outcomes = set()
    for depth in (8, 12):
        top = 2 * ((1 << depth) - 1)
        for width, height in ((64, 64), (61, 67), (40, 30), (33, 3), (5, 1), (1, 1)):
            n = width * height
            for back in (1, 2, 3, 4, 5, 9, 40, 200):
                if back > n:
                    continue
                for above in (0, 1, 2):
                    v = np.minimum(rng.integers(0, 3 << k, n), top)
                    v[n - back] = top + above
                    accepted = _check(_stream(v.astype(int).tolist(), k, depth, width, height))
                    assert accepted == (above == 0)
                    outcomes.add(accepted)
    assert outcomes == {True, False}
