"""Blocked differentiation of lattices of one row, one column and a few points:
every tile's region holds the lattice many times over, and the results are those
of the one-step kernels, bit for bit."""
import numpy as np
import pytest

import gmes_gb300 as G
from gmes_gb300.adjoint import DesignRegion

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny", [(1, 150), (150, 1), (2, 61), (61, 3), (5, 4)])
def test_thin_lattices(nx, ny):
    from gmes_gb300.adjoint import TMzAdjoint
    dx = 0.1

    def box(i, j, n, m):  # lattice points i .. i + n - 1, j .. j + m - 1
        return DesignRegion(center=((i + n / 2 - nx / 2) * dx, (j + m / 2 - ny / 2) * dx),
                            size=(n * dx, m * dx))

    i, j = nx // 2, ny // 2
    st = G.Continuous(freq=1.0, width=0.5)
    src = [G.PointSource(src_time=st, center=((i + .5 - nx / 2) * dx, (j + .5 - ny / 2) * dx, 0),
                         component=c) for c in (G.Jz, G.My)]
    design = box(min(i + 1, nx - 1), min(j + 1, ny - 1), 1, 1)
    monitor = box(max(i - 1, 0), max(j - 1, 0), 1, 1)
    out = []
    for block in (1, 4, 3):
        prob = TMzAdjoint(G.Cartesian(size=(nx * dx, ny * dx, 0), resolution=10),
                          [G.DefaultMedium(material=G.Dielectric())], src, design, monitor, 29,
                          batch=3, precision="fp32", block_steps=block)
        eps = np.array([2.0, 3.0, 5.0]).reshape(3, 1, 1) * np.ones((3,) + tuple(prob.shape))
        J = prob.forward(eps).cpu().numpy()
        g = prob.backward().cpu().numpy()
        out.append([J, g] + [prob.lattice(k).cpu().numpy() for k in range(3)]
                   + [prob.adjoint_field(k).cpu().numpy() for k in range(3)])
    assert out[0][0].min() > 0 and np.abs(out[0][1]).max() > 0
    for other in out[1:]:
        for k, (a, b) in enumerate(zip(out[0], other)):
            assert np.array_equal(a, b), k
