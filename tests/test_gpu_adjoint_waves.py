"""Blocked differentiation launches of about one block per SM.

While one block per SM holds a launch, its time is the slowest tile's, whatever
the batch; and a batch on either side of that line gives every design the values
that it has alone.
"""
import numpy as np
import pytest

import gmes_gb300 as G
from gmes_gb300.adjoint import DesignRegion

pytestmark = pytest.mark.gpu


def _problem(nx, ny, batch, steps=100):
    from gmes_gb300.adjoint import TMzAdjoint
    dx = 0.1
    geom = [G.DefaultMedium(material=G.Dielectric()),
            G.Shell(material=G.Cpml(), thickness=10 * dx)]
    src = [G.PointSource(src_time=G.Continuous(freq=1.0, width=1.0),
                         center=((14.5 - nx / 2) * dx, dx * q, 0), component=G.Jz)
           for q in range(-18, 19)]
    return TMzAdjoint(G.Cartesian(size=(nx * dx, ny * dx, 0), resolution=10), geom, src,
                      DesignRegion(center=(0, 0), size=(3.0, 3.0)),
                      DesignRegion(center=(2.0, 0), size=(0.3, 2.0)), steps, batch=batch,
                      precision="fp32", keep_history=True)


@pytest.mark.parametrize("batch", [14, 15, 16, 31])
def test_designs_do_not_depend_on_the_batch(batch):
    # 10 tiles per design: 140, 150, 160 and 310 blocks for 152 SMs
    eps = np.random.default_rng(2).uniform(1.0, 9.0, (batch, 30, 30))
    many, one = _problem(100, 100, batch, 61), _problem(100, 100, 1, 61)
    J, g = many.forward(eps).cpu().numpy(), many.backward().cpu().numpy()
    for b in (0, batch // 2, batch - 1):
        assert np.array_equal(one.forward(eps[b:b + 1]).cpu().numpy()[0], J[b])
        assert np.array_equal(one.backward().cpu().numpy()[0], g[b])
        assert np.abs(g[b]).max() > 0


def test_one_wave_takes_its_slowest_tile():
    import torch
    probs = {b: _problem(100, 100, b) for b in (4, 12)}
    took = {b: [] for b in probs}
    for _ in range(16):  # in turn: the clocks are the same for both
        for batch, prob in probs.items():
            eps = np.ones((batch, 30, 30))
            ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            prob.forward(eps)
            ev[0].record()
            prob.forward(eps)
            prob.backward()
            ev[1].record()
            torch.cuda.synchronize()
            took[batch].append(ev[0].elapsed_time(ev[1]))
    assert min(took[12]) < 1.1 * min(took[4]), took
