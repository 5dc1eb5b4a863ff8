"""The page-locked blocks that single-frame calls take their results from:
threads that end, threads that come one per call, calls at once."""

import threading

import pytest
import torch

import fastvid_b200
import oracle
from fastvid_b200 import synth
from fastvid_b200.codec import header_of

pytestmark = pytest.mark.gpu


def _frame(seed, cuda):
    planes = synth.make_frame(97 + seed, 61, "gray", 8, seed)
    kw = dict(layout="gray", bit_depth=8, quality=100, tile_size=(64, 64))
    return tuple(torch.from_numpy(p).to(cuda) for p in planes), kw, oracle.encode(planes, **kw)


def _round_trip(planes, kw, expected):
    stream = fastvid_b200.encode(planes, **kw)
    assert bytes(stream.cpu().numpy()) == expected
    assert torch.equal(fastvid_b200.decode(stream)[0].view(torch.int16), planes[0].view(torch.int16))


def test_a_thread_may_end_while_another_captures(cuda):
    frame = _frame(0, cuda)
    ready, go, failed = threading.Event(), threading.Event(), []

    def worker():
        try:
            with torch.cuda.stream(torch.cuda.Stream(cuda)):
                _round_trip(*frame)
                torch.cuda.current_stream().synchronize()
        except BaseException as e:
            failed.append(e)
        ready.set()
        go.wait(60)

    thread = threading.Thread(target=worker)
    thread.start()
    assert ready.wait(60) and not failed
    x = torch.zeros(8, device=cuda)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):  # global capture mode: unsafe calls of any thread end it
        x += 1
        go.set()
        thread.join(60)
        x += 1
    graph.replay()
    torch.cuda.synchronize()
    assert x.tolist() == [2.0] * 8
    _round_trip(*frame)


def test_a_thread_per_call_and_calls_at_once(cuda):
    frames = [_frame(seed, cuda) for seed in range(8)]
    failed = []

    def worker(frame, n):
        try:
            with torch.cuda.stream(torch.cuda.Stream(cuda)):
                for _ in range(n):
                    _round_trip(*frame)
        except BaseException as e:
            failed.append(e)

    for frame in frames:
        t = threading.Thread(target=worker, args=(frame, 1))
        t.start()
        t.join()
    threads = [threading.Thread(target=worker, args=(frame, 12)) for frame in frames]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failed, failed[0]


def test_a_header_read_is_a_thread_s_first_call(cuda):
    """A thread without a CUDA context of its own reads a header into a block
    that another thread left."""
    planes, kw, expected = _frame(3, cuda)
    stream = fastvid_b200.encode(planes, **kw)
    got = []
    for _ in range(3):
        t = threading.Thread(target=lambda: got.append(header_of(stream)))
        t.start()
        t.join()
    assert got == [expected[:32]] * 3
