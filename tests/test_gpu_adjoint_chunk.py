"""Differentiation with the steps of a call in one launch.

Small lattices take a call's steps in one cooperative launch, large ones two
launches per step.  The same designs in a small batch and among the many of a
large one must give bit-identical objective, fields and gradients, with
recorded history and with checkpoints; and so must a list of point sources
longer than the lattice map's places, in one-step and in blocked launches.
"""
import numpy as np
import pytest

import gmes_gb300 as G
from gmes_gb300.adjoint import DesignRegion

pytestmark = pytest.mark.gpu


def _args(nx, ny, hard=False, many=0, steps=37):
    dx = 0.1
    geom = [G.DefaultMedium(material=G.Dielectric()),
            G.Shell(material=G.Cpml(kappa_max=3.0), thickness=0.7)]
    st = G.Continuous(freq=1.0, width=1.0)
    src = [G.PointSource(src_time=st, center=(-0.7, dx * q, 0),
                         component=G.Ez if hard else G.Jz) for q in range(-6, 7)]
    src += [G.PointSource(src_time=st, center=(dx * (q % 40) - 1.98, dx * (q // 40) + 1.02, 0),
                          component=G.Jz) for q in range(many)]
    src += [G.PointSource(src_time=st, center=(0.4, 0.55, 0), component=G.Hx),
            G.PointSource(src_time=st, center=(0.45, -0.4, 0), component=G.My)]
    return (G.Cartesian(size=(nx * dx, ny * dx, 0), resolution=10), geom, src,
            DesignRegion(center=(0, 0), size=(0.9, 0.8)),
            DesignRegion(center=(0.3, -0.8), size=(0.3, 0.4)), steps)


def _run(args, eps, weight, **kw):
    from gmes_gb300.adjoint import TMzAdjoint
    prob = TMzAdjoint(*args, batch=eps.shape[0], courant_ratio=0.9, **kw)
    J = prob.forward(eps).cpu().numpy()
    state = [prob.lattice(k)[:2].cpu().numpy() for k in range(7)]
    g = prob.backward(weight).cpu().numpy()
    adj = [prob.adjoint_field(k)[:2].cpu().numpy() for k in range(3)]
    return prob, [J[:2], *state, g[:2], *adj]


@pytest.mark.parametrize("segment", [None, 8])
@pytest.mark.parametrize("precision,hard", [("fp64", False), ("fp64", True), ("df64", True),
                                            ("fp32", False)])
def test_one_launch_matches_launches_per_step(precision, hard, segment):
    nx, ny = 101, 131
    most = (1 << 20) if precision == "df64" else (1 << 22)
    args = _args(nx, ny, hard=hard)
    eps = np.random.default_rng(4).uniform(1.0, 9.0, (2, 9, 8))
    few, out = _run(args, eps, np.array([0.5, 1.5]), precision=precision, block_steps=1,
                    segment=segment)
    nb = most // (nx * ny) + 1
    many, want = _run(args, np.concatenate([eps, np.ones((nb - 2, 9, 8))]),
                      np.array([0.5, 1.5] + [1.0] * (nb - 2)), precision=precision,
                      block_steps=1, segment=segment)
    calls = 2 if segment is None else 3 * 5
    steps = args[-1] * (2 if segment is None else 3)
    assert few.launches() == 2 * calls and many.launches() == calls + 2 * steps
    assert np.isfinite(out[8]).all() and np.abs(out[8]).max() > 0 and out[0].min() > 0
    for k, (a, b) in enumerate(zip(out, want)):
        assert np.array_equal(a, b), k


def test_more_sources_than_places():
    args = _args(110, 126, many=1100)
    eps = np.random.default_rng(4).uniform(1.0, 9.0, (2, 9, 8))
    w = np.array([0.5, 1.5])
    prob, one = _run(args, eps, w, precision="fp32", block_steps=1)
    assert prob.desc.nsrc > 1023
    _, four = _run(args, eps, w, precision="fp32", block_steps=4)
    assert np.abs(one[8]).max() > 0
    for k, (a, b) in enumerate(zip(one, four)):
        assert np.array_equal(a, b), k


def test_block_steps_may_change_after_the_design_is_set():
    import ctypes as C

    from gmes_gb300 import _native as N
    from gmes_gb300.adjoint import TMzAdjoint
    args = _args(130, 140)
    eps = np.random.default_rng(4).uniform(1.0, 9.0, (2, 9, 8))
    prob = TMzAdjoint(*args, batch=2, precision="fp32", courant_ratio=0.9)
    prob.forward(eps)
    want = [prob.lattice(k).cpu().numpy() for k in range(7)]
    st = C.c_void_p(prob.grid.stream)
    prob.grid._enter()
    prob.design.fill_(0xab)  # nothing of the first design is left
    prob.grid._leave()
    prob.grid.synchronize()
    scratch, prob.desc.scratch, prob.desc.block_steps = prob.desc.scratch, None, 1
    prob._call("gmes_tmz_set_design", C.c_void_p(prob.eps.data_ptr()), st)
    prob.desc.scratch, prob.desc.block_steps = scratch, 4
    prob._call("gmes_tmz_reset", 1, st)
    prob._call("gmes_tmz_forward", 0, prob.nsteps, N.TMZ_RECORD_MONITOR, st)
    prob.grid.synchronize()
    assert np.abs(want[0]).max() > 0
    for k, w in enumerate(want):
        assert np.array_equal(prob.lattice(k).cpu().numpy(), w), k
