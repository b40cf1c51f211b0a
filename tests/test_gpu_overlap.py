"""Overlapped launches against calls that cannot overlap.

The kernels of one call come up while the one before them ends.  Whole arrays
of a call of many steps must equal those of the same half-steps as calls of
their own (whose first launch waits for everything before it), bit for bit: on
grids that keep the launches per half-step in each precision, with dispersive
media, complex fields and probes, in a batch, and for blocked differentiation
launches over tiles of every form.
"""
import numpy as np
import pytest

import gmes_gb300 as G
from test_gpu_adjoint_tiles import _problem
from test_gpu_persist import _scene, _start

pytestmark = pytest.mark.gpu

LARGE = dict(cls=G.FDTD, size=(5.4, 5.2, 5.0))  # above 2^17 cells
CASES = {
    "cube_fp64": (dict(LARGE, edge=True), "fp64"),
    "cube_fp32": (dict(LARGE, edge=True), "fp32"),
    "cube_df64": (dict(LARGE, kappa=3.0), "df64"),
    "cube_strict": (dict(cls=G.FDTD, size=(2.4, 2.2, 2.1)), "fp64_strict"),
    "dcp_upml_fp64": (dict(LARGE, medium="dcp", pml="upml"), "fp64"),
    "drude_fp32": (dict(LARGE, medium="drude"), "fp32"),
    "bloch": (dict(cls=G.FDTD, size=(6.6, 6.4, 6.3), bloch=(0.4, -0.3, 0.2)), "fp64"),
}


def _half_steps(e, n0, k):
    e.stage_sources(float(n0), k)
    for s in range(k):
        e.half_step(0, s)
        e.half_step(1, s)
    e.synchronize()


def _assert_same(a, b):
    for c in range(6):
        fa, fb = a.fields[c].cpu().numpy(), b.fields[c].cpu().numpy()
        assert np.isfinite(fa).all()
        assert np.array_equal(fa, fb), c
        if a.aux[c] is not None:
            assert np.array_equal(a.aux[c].cpu().numpy(), b.aux[c].cpu().numpy()), c


@pytest.mark.parametrize("name", list(CASES))
def test_call_equals_half_step_calls(name):
    kw, precision = CASES[name]
    a = _start(_scene(res=10, precision=precision, **kw))
    b = _start(_scene(res=10, precision=precision, **kw))
    assert a.step_launches(17) > 17
    n = 0
    for k in (1, 2, 17):
        a.step(k, n0=float(n))
        a.synchronize()
        _half_steps(b, n, k)
        _assert_same(a, b)
        n += k


def test_probes_see_the_fields_of_their_step():
    def make():
        e = _start(_scene(G.TMzFDTD, (20.1, 14.3, 0), 10, "fp64"))
        e.set_probes([(2, 71 * 144 + 33), (3, 2 * 3000 + 17), (4, 9001)])
        return e
    a, b = make(), make()
    a.step(11)
    got = a.probe_values(11)
    for s in range(11):
        b.step(1, n0=float(s))
        assert np.array_equal(b.probe_values(1)[0], got[s])
    assert np.abs(got).max() > 0


@pytest.mark.parametrize("precision", ["fp64", "fp32", "df64"])
def test_batch_equals_half_step_calls(precision):
    from gmes_gb300.batch import Batch
    kws = [dict(cls=G.FDTD, size=(4.4, 4.7, 4.1)), dict(cls=G.TMzFDTD, size=(9.1, 20.3, 0)),
           dict(cls=G.FDTD, size=(3.1, 2.9, 3.3), medium="drude"),
           dict(cls=G.TEzFDTD, size=(12.3, 6.5, 0), comp=G.Jx)]
    a = [_start(_scene(res=10, precision=precision, **kw)) for kw in kws]
    b = [_start(_scene(res=10, precision=precision, **kw)) for kw in kws]
    batch = Batch(a, solo_cells=0)
    steps = [13, 13, 9, 13]
    batch.run(steps, [0.0] * 4)
    batch.synchronize()
    for x, y, k in zip(a, b, steps):
        x.synchronize()
        _half_steps(y, 0, k)
        _assert_same(x, y)


def test_blocked_launches_over_every_tile_form():
    from gmes_gb300.adjoint import TMzAdjoint
    args, eps = _problem(260, 381, batch=6, pml="two", strip=True, hsrc=True, hard=True,
                         design=(40, 60), steps=61)
    out = []
    for block in (1, 4):
        prob = TMzAdjoint(*args, batch=6, precision="fp32", block_steps=block, courant_ratio=0.9)
        J = prob.forward(eps).cpu().numpy()
        g = prob.backward().cpu().numpy()
        out.append([J, g] + [prob.lattice(k).cpu().numpy() for k in range(7)]
                   + [prob.adjoint_field(k).cpu().numpy() for k in range(3)])
    assert np.abs(out[0][1]).max() > 0
    for k, (x, y) in enumerate(zip(*out)):
        assert np.array_equal(x, y), k
