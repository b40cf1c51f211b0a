"""A one-launch step whose wait runs out.

A block that stays away from a barrier makes the others give up after a few
polls.  What meets at that slot afterwards gives up at once: stepped fields,
objective and gradient read as NaN, calls that wait or step raise, and after a
reset everything works as before.  Nothing waits longer than the polls given.
"""
import ctypes as C

import numpy as np
import pytest

import gmes_gb300 as G
from gmes_gb300 import _native as N
from test_gpu_adjoint_chunk import _args
from test_gpu_persist import _scene, _start

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def _cleared():
    yield
    N.clear_waits()


def _check(stream, absent, blocks=5, polls=40):
    import torch
    out = torch.zeros(1001, dtype=torch.float64, device="cuda")
    with torch.cuda.stream(torch.cuda.ExternalStream(stream)):
        torch.cuda._sleep(int(3e7))  # so that what follows is enqueued before the wait
    N.check(N.load().gmes_wait_check(blocks, absent, polls, C.c_void_p(out.data_ptr()),
                                     out.numel() * 8, C.c_void_p(stream)))
    return out


@pytest.mark.parametrize("absent", [0, 2, 4])
def test_wait_runs_out(absent):
    import torch
    s = torch.cuda.Stream()
    fine = _check(s.cuda_stream, -1, polls=1 << 20)
    s.synchronize()
    N.check_waits()
    assert not fine.cpu().numpy().any()
    out = _check(s.cuda_stream, absent)
    s.synchronize()
    with pytest.raises(RuntimeError, match="gave up"):
        N.check_waits()
    left = out.cpu().numpy()
    # the absent block's share alone is untouched
    assert np.isnan(left).any() and np.isfinite(left).sum() <= 1001 // 5 + 32
    N.clear_waits()
    N.check_waits()
    again = _check(s.cuda_stream, -1, polls=1 << 20)
    s.synchronize()
    N.check_waits()
    assert not again.cpu().numpy().any()


def test_step_after_a_wait_that_ran_out():
    e, other, want = (_start(_scene(G.TMzFDTD, (6.1, 4.3, 0), 10, "fp64")) for _ in range(3))
    e.use_graphs = False
    e.step(3)
    e.synchronize()
    graph = other._graph(3)
    for x in (e, other, want):
        x.stage_sources(0.0, x.src_chunk)
        x.synchronize()
    _check(e.stream, 1)
    e.launch_raw(3)  # enqueued before the wait ran out
    e._stream.synchronize()
    with pytest.raises(RuntimeError, match="gave up"):
        e.synchronize()
    with pytest.raises(RuntimeError, match="gave up"):
        e.read(2)
    with pytest.raises(RuntimeError, match="gave up"):
        e.step(1)
    with pytest.raises(RuntimeError, match="gave up"):
        other.launch_raw(3)
    for c in (2, 3, 4):
        assert np.isnan(e.fields[c].cpu().numpy()).all()
    N.clear_waits()
    assert graph == other._graph(3)
    other.launch_raw(3)
    want.use_graphs = False
    want.launch_raw(3)
    for c in (2, 3, 4):
        assert np.array_equal(other.read(c), want.read(c))
        assert np.isfinite(want.read(c)).all()


def test_batches_after_a_wait_that_ran_out():
    import torch

    from gmes_gb300.batch import Batch
    grids = [_start(_scene(G.FDTD, (1.9, 1.7, 1.6), 10, "fp64")) for _ in range(3)]
    alone = grids.pop()
    batch = Batch(grids, use_graphs=False)
    batch.run([2, 2], [0.0, 0.0])
    batch.synchronize()
    s = torch.cuda.Stream()
    _check(s.cuda_stream, 0)
    s.synchronize()
    with pytest.raises(RuntimeError, match="gave up"):
        batch.run([2, 2], [2.0, 2.0])
    with pytest.raises(RuntimeError, match="gave up"):
        batch.synchronize()
    N.clear_waits()
    batch.run([2, 2], [2.0, 2.0])
    batch.synchronize()
    alone.step(2)
    alone.step(2, n0=2.0)
    for e in grids:  # untouched by the other launch
        for c in range(6):
            assert np.array_equal(e.read(c), alone.read(c))


@pytest.mark.parametrize("segment", [None, 8])
def test_differentiation_after_a_wait_that_ran_out(segment):
    from gmes_gb300.adjoint import TMzAdjoint
    args = _args(60, 61, steps=19)
    eps = np.random.default_rng(4).uniform(1.0, 9.0, (2, 9, 8))
    prob = TMzAdjoint(*args, batch=2, precision="fp64", courant_ratio=0.9, segment=segment)
    want = [prob.forward(eps).cpu().numpy(), prob.backward().cpu().numpy()]
    N.check_waits()
    _check(prob.grid.stream, 1)
    J = prob.forward(eps)  # forward and backward enqueued before the wait ran out, or refused
    try:
        g = prob.backward()
    except RuntimeError as error:
        assert "gave up" in str(error)
        g = None
    prob.grid._stream.synchronize()
    assert np.isnan(J.cpu().numpy()).all()
    assert g is None or np.isnan(g.cpu().numpy()).all()
    with pytest.raises(RuntimeError, match="gave up"):
        prob.lattice(0)
    with pytest.raises(RuntimeError, match="gave up"):
        prob.forward(eps)
    N.clear_waits()
    got = [prob.forward(eps).cpu().numpy(), prob.backward().cpu().numpy()]
    for a, b in zip(got, want):
        assert np.array_equal(a, b)


def test_bad_arguments():
    lib = N.load()
    for blocks, absent, polls in ((0, -1, 9), (100000, -1, 9), (4, 4, 9), (4, -2, 9), (4, 0, 0),
                                  (4, 0, 1 << 30)):
        with pytest.raises(ValueError):
            N.check(lib.gmes_wait_check(blocks, absent, polls, None, 0, None))
    with pytest.raises(ValueError):
        N.check(lib.gmes_wait_check(4, -1, 9, None, 8, None))
