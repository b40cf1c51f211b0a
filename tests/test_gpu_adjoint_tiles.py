"""The tile forms of the temporally blocked differentiation kernels.

A blocked launch treats each tile by what its points are: plain, absorbing
rows, columns or both, special points (sources, monitor, design pixels) and a
per-point form for the rest.  Against the one-step kernels, objective, fields,
psi and gradients must be bit-identical on scenes that make every form: an odd
lattice, a dielectric strip that runs into the absorbing layer, two layers, a
layer on two sides only, a source of an H component, hard sources, a design
region that reaches over several tiles and next to the layer, and one row.
"""
import numpy as np
import pytest

import gmes_gb300 as G
from gmes_gb300.adjoint import DesignRegion

pytestmark = pytest.mark.gpu


def _problem(nx, ny, batch=2, pml="one", strip=False, hsrc=False, hard=False, design=(9, 8),
             shift=(0.0, 0.0), steps=46):
    dx = 0.1
    geom = [G.DefaultMedium(material=G.Dielectric())]
    if strip:
        geom.append(G.Block(material=G.Dielectric(eps_inf=3.0), center=(0, 0.9, 0),
                            size=(2 * nx * dx, 0.6, 1)))
    if pml == "one":
        geom.append(G.Shell(material=G.Cpml(kappa_max=3.0), thickness=0.7))
    elif pml == "two":
        geom.append(G.Shell(material=G.Cpml(), thickness=0.9))
        geom.append(G.Shell(material=G.Cpml(m=3.0), thickness=0.4))
    elif pml == "sides":
        geom.append(G.Shell(material=G.Cpml(), thickness=0.8, plus_y=False, minus_y=False))
    st = G.Continuous(freq=1.0, width=1.0)
    x_src = shift[0] - (0.7 if nx < 60 else 1.0)  # the wave reaches design and monitor
    src = [G.PointSource(src_time=st, center=(x_src, shift[1] + dx * q, 0),
                         component=G.Ez if hard else G.Jz) for q in range(-6, 7)]
    if hsrc:
        src.append(G.PointSource(src_time=st, center=(0.4, 0.55, 0), component=G.Hx))
        src.append(G.PointSource(src_time=st, center=(0.45, -0.4, 0), component=G.My))
    space = G.Cartesian(size=(nx * dx, ny * dx, 0), resolution=10)
    des = DesignRegion(center=shift, size=(design[0] * dx, design[1] * dx))
    mon = DesignRegion(center=(shift[0] + 0.3, shift[1] - 0.8), size=(0.3, 0.4))
    eps = np.random.default_rng(4).uniform(1.0, 9.0, (batch,) + tuple(design))
    return (space, geom, src, des, mon, steps), eps


CASES = {
    "even_130x190": dict(nx=130, ny=190),
    "odd_101x131": dict(nx=101, ny=131, design=(31, 40)),
    "strip_into_layer": dict(nx=96, ny=120, strip=True),
    "two_layers": dict(nx=90, ny=119, pml="two"),
    "two_sides": dict(nx=90, ny=125, pml="sides"),
    "no_layer": dict(nx=75, ny=70, pml="none"),
    "h_sources": dict(nx=90, ny=126, hsrc=True),
    "hard_sources": dict(nx=90, ny=127, hard=True),
    "design_at_layer": dict(nx=88, ny=120, shift=(-2.0, 4.0), design=(14, 20)),
    "narrow": dict(nx=34, ny=300, steps=43),
}


@pytest.mark.parametrize("name", list(CASES))
def test_tile_forms_match_one_step_kernels(name):
    from gmes_gb300.adjoint import TMzAdjoint
    args, eps = _problem(**CASES[name])
    out = []
    for steps in (1, 4, 3):
        prob = TMzAdjoint(*args, batch=eps.shape[0], precision="fp32", block_steps=steps,
                          courant_ratio=0.9)
        J = prob.forward(eps).cpu().numpy()
        state = [prob.lattice(k).cpu().numpy() for k in range(7)]
        g = prob.backward(np.linspace(0.5, 1.5, eps.shape[0])).cpu().numpy()
        adj = [prob.adjoint_field(k).cpu().numpy() for k in range(3)]
        out.append((J, state, g, adj))
    J1, s1, g1, a1 = out[0]
    assert np.isfinite(g1).all() and np.abs(g1).max() > 0 and J1.min() > 0
    for J, s, g, a in out[1:]:
        assert np.array_equal(J, J1)
        for k in range(7):
            assert np.array_equal(s[k], s1[k]), k
        assert np.array_equal(g, g1)
        for k in range(3):
            assert np.array_equal(a[k], a1[k]), k
