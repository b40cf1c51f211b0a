"""Cooperative launches in flight together never meet at one barrier slot.

A launch queued behind other work on one stream while more than a thousand
calls pass on another; several threads with a stream each; and graphs that the
caller captures, replays and destroys.  Fields must equal those of the same
steps made one after another.
"""
import ctypes as C
import threading

import numpy as np
import pytest

import gmes_gb300 as G
from gmes_gb300 import _native as N
from test_gpu_persist import _scene, _start

pytestmark = pytest.mark.gpu


def _engine(size=(6.1, 4.3, 0)):
    return _start(_scene(G.TMzFDTD, size, 10, "fp64"))


def _direct(e, stream, k):
    N.check(e.lib.gmes_step(C.byref(e.desc), k, C.c_void_p(stream.cuda_stream)))


def _fields(e):
    return [f.cpu().numpy() for f in e.fields if f is not None]


def _same(a, b):
    a, b = _fields(a), _fields(b)
    assert all(np.isfinite(x).all() for x in a) and max(np.abs(x).max() for x in a) > 0
    return all(np.array_equal(x, y) for x, y in zip(a, b))


def test_queued_launch_and_a_thousand_calls():
    import torch
    queued, other, want_q, want_o = _engine(), _engine(), _engine(), _engine()
    for e in (queued, other, want_q, want_o):
        e.stage_sources(0.0, e.src_chunk)
        e.synchronize()
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(s1):
        torch.cuda._sleep(int(3e7))  # some 15 ms
    _direct(queued, s1, 40)
    for _ in range(1100):
        _direct(other, s2, 1)
    _direct(queued, s1, 3)
    torch.cuda.synchronize()
    s3 = torch.cuda.Stream()
    _direct(want_q, s3, 40)
    _direct(want_q, s3, 3)
    torch.cuda.synchronize()
    for _ in range(1100):
        _direct(want_o, s3, 1)
        torch.cuda.synchronize()
    assert _same(queued, want_q) and _same(other, want_o)


def test_threads_with_a_stream_each():
    import torch
    engines, want = [_engine() for _ in range(4)], _engine()
    streams = [torch.cuda.Stream() for _ in engines]
    for e in engines + [want]:
        e.stage_sources(0.0, e.src_chunk)
        e.synchronize()

    def work(e, s):
        for k in (1, 5, 2) * 60:
            _direct(e, s, k)

    th = [threading.Thread(target=work, args=p) for p in zip(engines, streams)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    torch.cuda.synchronize()
    work(want, streams[0])
    torch.cuda.synchronize()
    assert all(_same(e, want) for e in engines)


def test_captures_of_the_caller():
    import torch
    e, want = _engine(), _engine()
    for x in (e, want):
        x.stage_sources(0.0, x.src_chunk)
        x.synchronize()
    s = torch.cuda.Stream()
    _direct(want, s, 1)  # loads the kernels before any capture
    torch.cuda.synchronize()
    for _ in range(5):
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            _direct(e, s, 7)
            _direct(e, s, 2)
        g.replay()
        g.replay()
        del g  # possibly in flight
    torch.cuda.synchronize()
    want2 = _engine()
    want2.stage_sources(0.0, want2.src_chunk)
    want2.synchronize()
    for _ in range(10):
        _direct(want2, s, 7)
        _direct(want2, s, 2)
    torch.cuda.synchronize()
    assert _same(e, want2)
