"""One-launch steps without their shared-memory tables: short calls and large grids.

A call of a few steps builds no tables and must not be slower than the
half-step launches that it replaces; a grid whose tables do not fit does
without them in calls of any length, with the same values.
"""
import numpy as np
import pytest

import gmes_gb300 as G
from test_gpu_overlap import _assert_same, _half_steps
from test_gpu_persist import _scene, _start

pytestmark = pytest.mark.gpu

LARGE = {
    "tmz_fp64": (dict(cls=G.TMzFDTD, size=(103.0, 102.7, 0), edge=True), "fp64"),
    "tmz_fp32": (dict(cls=G.TMzFDTD, size=(113.0, 112.7, 0), kappa=3.0), "fp32"),
    "tez_drude_df64": (dict(cls=G.TEzFDTD, size=(90.1, 121.3, 0), medium="drude", comp=G.Jx),
                       "df64"),
    "row_fp32": (dict(cls=G.TMzFDTD, size=(4.1, 400.3, 0), pml="none"), "fp32"),
    "bloch": (dict(cls=G.TEzFDTD, size=(103.1, 102.3, 0), bloch=(0.4, -0.3, 0), pml="none",
                   comp=G.Jx), "fp64"),
}


@pytest.mark.parametrize("name", list(LARGE))
def test_grids_beyond_the_tables(name):
    kw, precision = LARGE[name]
    a = _start(_scene(res=10, precision=precision, **kw))
    b = _start(_scene(res=10, precision=precision, **kw))
    assert a.step_launches(6) == 1
    a.step(6)
    a.synchronize()
    _half_steps(b, 0, 6)
    _assert_same(a, b)


@pytest.mark.parametrize("size,precision", [((3.2, 3.2, 3.2), "df64"), ((3.2, 3.2, 3.2), "fp32"),
                                            ((90.0, 90.0, 0), "fp32"), ((6.4, 6.4, 0), "df64")])
def test_one_step_calls_are_no_slower(size, precision):
    import torch
    cls = G.FDTD if size[2] else G.TMzFDTD
    e = _start(_scene(cls, size, 10, precision))
    assert e.step_launches(1) == 1
    e.stage_sources(0.0, 1)
    e.use_graphs = False
    s = e.torch_stream

    def halves():
        e.half_step(0, 0)
        e.half_step(1, 0)

    graphs = {}
    for name, step in (("one", lambda: e.launch_raw(1)), ("halves", halves)):
        step()
        torch.cuda.synchronize()
        graphs[name] = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graphs[name], stream=s):
            for _ in range(20):
                step()
    took = {name: [] for name in graphs}
    for _ in range(12):  # in turn: the clocks are the same for both
        for name, graph in graphs.items():
            ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            graph.replay()
            ev[0].record()
            graph.replay()
            graph.replay()
            ev[1].record()
            torch.cuda.synchronize()
            took[name].append(ev[0].elapsed_time(ev[1]))
    assert min(took["one"]) < 0.97 * min(took["halves"]), took
    assert all(np.isfinite(f.cpu().numpy()).all() for f in e.fields if f is not None)
