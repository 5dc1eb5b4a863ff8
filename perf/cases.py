"""Performance cases: the codec calls that users of this framework make.

Every case is one call of the public API -- ``fastvid_b200.api`` for one
frame, ``fastvid_b200.batch`` for a list -- on planes or streams that are
already on the GPU.  The caller keeps its output buffer, as a recorder or a
player does: a list's streams or planes go straight into it (``arena``), a
single frame's stream is copied into it.  Frames are seeded
synthetic pictures made on the GPU: sinusoid layers with periods of 32 to 256
pixels, rectangles with sharp edges and Gaussian noise, every fourth frame of
a list near-flat.  Sizes, formats, qualities and tile sizes are those of the
benchmark mix, the serving mix, the evaluator's gates and the API defaults.

All outputs are whole numbers (stream bytes, plane samples), equal on every
run, so there are no 64-bit reference values.
"""

from __future__ import annotations

import math

import torch

from fastvid_b200 import api, batch

# the serving and benchmark mixes' formats: (share, width, height, layout, depth, quality, tile, noise sd)
_MIX = (
    (2, 1280, 720, "gray", 8, 100, 64, 3.0),
    (2, 1920, 1080, "rgb444", 8, 90, 128, 3.0),
    (1, 3840, 2160, "rgb444", 10, 85, 128, 4.0),
    (1, 2048, 1080, "gray", 16, 87, 128, 40.0),
)
_MIX_SHARES = sum(m[0] for m in _MIX)


def _case(op, width, height, layout, depth, quality, tile_w, tile_h, noise, count=0):
    """count 0: one frame through the single-frame call; n: a list of n frames."""
    return dict(op=op, width=width, height=height, layout=layout, depth=depth, quality=quality, tile_w=tile_w,
                tile_h=tile_h, noise=noise, count=count)


def listed():
    cases = [
        # a thumbnail or a preview tile: the smallest calls, launches and host work count
        dict(_case("encode", 320, 180, "gray", 8, 100, 256, 128, 3.0), name="encode_thumb_gray8"),
        dict(_case("decode", 320, 180, "gray", 8, 100, 256, 128, 3.0), name="decode_thumb_gray8"),
        # one 720p luma frame with the benchmark mix's small tiles (a camera or a mask channel, lossless)
        dict(_case("encode", 1280, 720, "gray", 8, 100, 64, 64, 3.0), name="encode_720p_gray8"),
        # the latency gates: one 1080p RGB frame with the API's default tiles
        dict(_case("encode", 1920, 1080, "rgb444", 8, 90, 256, 128, 3.0), name="encode_1080p_rgb8"),
        dict(_case("decode", 1920, 1080, "rgb444", 10, 90, 256, 128, 4.0), name="decode_1080p_rgb10"),
        # a crop of odd size in subsampled 12-bit video: ragged tiles, planes and shards
        dict(_case("decode", 1437, 811, "yuv422", 12, 95, 256, 128, 16.0), name="decode_odd_yuv422_12"),
        # one 4K 16-bit frame: the encoder's refined-step trial is a second pass
        dict(_case("encode", 3840, 2160, "gray", 16, 87, 128, 128, 40.0), name="encode_4k_gray16"),
        # an archive frame, 16-bit lossless: symbols wider than 16 bits
        dict(_case("decode", 3840, 2160, "gray", 16, 100, 128, 128, 40.0), name="decode_4k_gray16_lossless"),
        # the throughput gates: a second of 4K video encoded, and a shot decoded, as one list
        dict(_case("encode", 3840, 2160, "yuv422", 10, 90, 256, 128, 4.0, count=24), name="encode_24x4k_yuv422_10"),
        dict(_case("decode", 3840, 2160, "rgb444", 10, 90, 256, 128, 4.0, count=16), name="decode_16x4k_rgb10"),
        # a server's or an ingest job's batch of mixed formats
        dict(_case("encode", 0, 0, "mixed", 0, 0, 0, 0, 0.0, count=18), name="encode_mixed_18"),
        dict(_case("decode", 0, 0, "mixed", 0, 0, 0, 0, 0.0, count=18), name="decode_mixed_18"),
    ]
    return cases


def _samples(layout, width, height):
    if layout == "gray":
        return width * height
    if layout == "rgb444":
        return 3 * width * height
    return (width + 2 * ((width + 1) // 2)) * height


def draw(rng):
    """A case of the same ranges: any layout and depth, qualities from coarse
    to lossless, frames from 160x90 to 4K of odd and even sizes, tiles of the
    API default and the tuning table, single frames and lists."""
    op = rng.choice(("encode", "decode"))
    if rng.random() < 0.15:
        return _case(op, 0, 0, "mixed", 0, 0, 0, 0, 0.0, count=rng.randint(6, 18))
    layout = rng.choice(("gray", "yuv422", "rgb444"))
    depth = rng.choice((8, 10, 12, 16))
    quality = rng.choice((100, 100, 96, 90, 90, 87, 85, 66, 50))
    width = int(round(math.exp(rng.uniform(math.log(160), math.log(3840)))))
    height = max(90, min(2160, int(round(width * rng.uniform(0.5, 0.8)))))
    if rng.random() < 0.5:  # half of the frames of even sizes, as video mostly has
        width, height = width & ~7, height & ~1
    tile_w, tile_h = rng.choice(((256, 128), (256, 128), (128, 128), (64, 64)))
    noise = {8: 3.0, 10: 4.0, 12: 16.0, 16: 40.0}[depth] * rng.choice((0.25, 1.0, 1.0, 2.0))
    count = 0
    if rng.random() < 0.5:
        most = max(2, min(16, 130_000_000 // _samples(layout, width, height)))
        count = int(round(math.exp(rng.uniform(math.log(2), math.log(most)))))
    return _case(op, width, height, layout, depth, quality, tile_w, tile_h, noise, count)


def _frame(width, height, layout, depth, noise, flat, gen):
    """One frame's planes (uint16, on the GPU)."""
    maximum = (1 << depth) - 1
    amplitude = 20000.0 if depth == 16 else 60.0 * (maximum + 1) / 256.0
    dev = gen.device

    def uniform(n):
        return torch.rand(n, generator=gen, device=dev, dtype=torch.float64).cpu().tolist()

    def field(w):
        u = uniform(12)
        y = torch.arange(height, device=dev, dtype=torch.float32)[:, None]
        x = torch.arange(w, device=dev, dtype=torch.float32)[None, :]
        total = sum(u[0:4]) + 1e-9
        out = torch.zeros(height, w, device=dev)
        for i in range(4):
            period = 32.0 * 8.0 ** u[4 + i]
            angle = 2 * math.pi * u[8 + i]
            kx, ky = 2 * math.pi / period * math.cos(angle), 2 * math.pi / period * math.sin(angle)
            out += torch.sin(x * kx + y * ky + 6.0 * u[i]) * (amplitude * u[i] / total)
        return out

    half = layout == "yuv422"
    widths = [width] if layout == "gray" else [width] + [(width + 1) // 2 if half else width] * 2
    shared = field(width) if layout == "rgb444" else None
    planes = []
    for w in widths:
        p = field(w)
        if shared is not None:
            p = 0.8 * shared + 0.6 * p
        p += (maximum + 1) / 2
        u = uniform(50)
        for i in range(10):
            rw, rh = max(1, int(w / 16 + u[5 * i] * w / 5)), max(1, int(height / 16 + u[5 * i + 1] * height / 5))
            x0, y0 = int(u[5 * i + 2] * (w - rw)), int(u[5 * i + 3] * (height - rh))
            p[y0:y0 + rh, x0:x0 + rw] = round(u[5 * i + 4] * maximum)
        p += torch.randn(height, w, generator=gen, device=dev) * (0.5 if flat else noise)
        planes.append(p.round_().clamp_(0, maximum).to(torch.int32).to(torch.uint16))
    return tuple(planes)


def _formats(case):
    """(width, height, layout, depth, quality, (tile_w, tile_h), noise) of each frame of a case."""
    if case["layout"] != "mixed":
        one = (case["width"], case["height"], case["layout"], case["depth"], case["quality"],
               (case["tile_w"], case["tile_h"]), case["noise"])
        return [one] * max(1, case["count"])
    out = []
    for share, w, h, layout, depth, quality, tile, noise in _MIX:
        out += [(w, h, layout, depth, quality, (tile, tile), noise)] * max(1, case["count"] * share // _MIX_SHARES)
    return out


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    formats = _formats(case)
    frames = [_frame(w, h, layout, depth, noise, len(formats) > 1 and i % 4 == 3, gen)
              for i, (w, h, layout, depth, _, _, noise) in enumerate(formats)]
    state = {"op": case["op"], "list": case["count"] > 0, "input": frames}
    samples = sum(p.numel() for f in frames for p in f)
    if state["list"]:
        state["params"] = dict(layout=[f[2] for f in formats], bit_depth=[f[3] for f in formats],
                               quality=[f[4] for f in formats], tile_size=[f[5] for f in formats])
    else:
        state["params"] = dict(format=case["layout"], bit_depth=case["depth"], quality=case["quality"],
                               tile_size=(case["tile_w"], case["tile_h"]))
        state["input"] = frames[0]
    if case["op"] == "decode":
        if state["list"]:
            # copies of their own: streams as read from files or the network
            state["input"] = [s.clone() for s in batch.encode_batch(frames, **state["params"])]
            state["arena"] = torch.zeros(samples, dtype=torch.uint16, device=gen.device)
        else:
            state["input"] = api.encode(frames[0], **state["params"])
    else:
        # room for any content: 17 bits a sample, the directory and the record headers
        state["arena"] = torch.zeros(samples * 17 // 8 + samples // 64 + 65536 * len(formats), dtype=torch.uint8,
                                     device=gen.device)
    return state


def run(state):
    if state["op"] == "encode":
        arena = state["arena"]
        if state["list"]:
            streams = batch.encode_batch(state["input"], arena=arena, **state["params"])
            return {"arena": arena, "lengths": [s.numel() for s in streams]}
        stream = api.encode(state["input"], **state["params"])
        arena[:stream.numel()].copy_(stream)
        return {"arena": arena, "lengths": [stream.numel()]}
    # planes as int16, the same bits
    if state["list"]:
        arena = state["arena"]
        batch.default_codec(arena.device).decode(state["input"], arena=arena)
        return arena.view(torch.int16)
    return [p.view(torch.int16) for p in api.decode(state["input"])]


def _step(layout, depth, quality):
    if depth == 8 and layout != "rgb444":
        return 1
    den = {("yuv422", 10): 20, ("yuv422", 16): 24, ("rgb444", 10): 10}.get((layout, depth), 6)
    return 1 + ((100 - quality) * (1 << (depth - 8)) + den - 1) // den


def work(case):
    """Encode: planes in, stream out; decode: stream in, planes out.  The
    stream's size is estimated from the noise: the prediction residual of
    white noise of deviation s is about 1.7 s, quantized by the step."""
    total = 0.0
    formats = _formats(case)
    for i, (w, h, layout, depth, quality, _, noise) in enumerate(formats):
        n = _samples(layout, w, h)
        sd = 1.7 * (0.5 if len(formats) > 1 and i % 4 == 3 else noise) / _step(layout, depth, quality)
        bits = max(0.1, 0.5 * math.log2(2 * math.pi * math.e * (sd * sd + 0.05)))
        total += n * (2 + bits / 8)
    return {"bytes": total, "flops": 0.0}


def exact(case, seed):
    return None
