"""Long lists of point sources in one-step differentiation.

Short lists are looked up by the points' bodies, long ones walked entry by entry:
by the blocks of a one-launch call, each for its own points (also when a block
has more of them than it can note), and in launches of their own.  All must agree
bit for bit, with E and H sources on the same points, hard and current, and
with the FP32 blocked launches; and a long list must not cost much more than a
short one.
"""
import numpy as np
import pytest

import gmes_gb300 as G
from gmes_gb300 import _native as N
from gmes_gb300.adjoint import DesignRegion
from test_gpu_adjoint_chunk import _args

pytestmark = pytest.mark.gpu


def _problem(nx, ny, batch, rows, vals, precision, steps, **kw):
    """A problem whose source list is replaced by rows (comp, mode, offset)."""
    import torch
    from gmes_gb300.adjoint import TMzAdjoint
    args = list(_args(nx, ny, steps=steps))
    args[4] = DesignRegion(center=(0.3, 0.6), size=(0.5, 0.8))
    prob = TMzAdjoint(*args, batch=batch, precision=precision, courant_ratio=0.9, **kw)
    arr = (N.PointSourceC * len(rows))(*[N.PointSourceC(c, m, o) for c, m, o in rows])
    prob.src = torch.frombuffer(bytearray(bytes(arr)), dtype=torch.uint8).to(prob.device)
    prob.src_val = torch.from_numpy(np.ascontiguousarray(vals)).to(prob.device)
    prob.desc.nsrc = len(rows)
    prob.desc.src = prob.src.data_ptr()
    prob.desc.src_val = prob.src_val.data_ptr()
    torch.cuda.synchronize()
    return prob


def _list(nx, ny, n, seed=5, hard=True):
    """n entries of distinct (component, point), half the points with an E and H entry."""
    rng = np.random.default_rng(seed)
    at = rng.permutation(nx * ny)[:(2 * n + 2) // 3]
    rows = [(2, int(hard and rng.random() < 0.3), int(o)) for o in at]
    rows += [(int(rng.integers(3, 5)), int(hard and rng.random() < 0.3), int(o)) for o in at]
    rows = [(c, 1 - m, o) for c, m, o in rows[:n]]  # mode 0: hard
    rows += [(2, 1, -1), (3, 0, nx * ny), (1, 1, 3)]  # name no point: skipped
    return rows


def _run(prob, eps, weight):
    J = prob.forward(eps).cpu().numpy()
    state = [prob.lattice(k)[:2].cpu().numpy() for k in range(7)]
    g = prob.backward(weight).cpu().numpy()
    adj = [prob.adjoint_field(k)[:2].cpu().numpy() for k in range(3)]
    return [J[:2], *state, g[:2], *adj]


@pytest.mark.parametrize("n", [28, 29, 30, 61, 700])
@pytest.mark.parametrize("precision", ["fp64", "df64", "fp32"])
def test_routes_agree(precision, n):
    nx, ny, steps = 101, 131, 9
    rows = _list(nx, ny, n)
    vals = np.random.default_rng(6).standard_normal((steps, 2, len(rows)))
    eps = np.random.default_rng(4).uniform(1.0, 9.0, (2, 9, 8))
    weight = np.array([0.5, 1.5])
    one = _problem(nx, ny, 2, rows, vals, precision, steps, block_steps=1, segment=4)
    out = _run(one, eps, weight)
    assert all(np.isfinite(x).all() for x in out) and np.abs(out[8]).max() > 0
    most = (1 << 20) if precision == "df64" else (1 << 22)
    nb = most // (nx * ny) + 1
    many = _problem(nx, ny, nb, rows, vals, precision, steps, block_steps=1, segment=4)
    wants = [_run(many, np.concatenate([eps, np.ones((nb - 2, 9, 8))]),
                  np.array([0.5, 1.5] + [1.0] * (nb - 2)))]
    calls, walked = 3 * 3, len(rows) > 32
    assert one.launches() == calls * (1 if walked else 2)
    assert many.launches() == (4 * 3 * steps if walked else calls + 2 * 3 * steps)
    if precision == "fp32":
        wants.append(_run(_problem(nx, ny, 2, rows, vals, precision, steps, block_steps=4), eps,
                          weight))
    for want in wants:
        for k, (a, b) in enumerate(zip(out, want)):
            assert np.array_equal(a, b), k


def test_more_entries_than_a_block_notes():
    nx, ny, nb, steps = 200, 250, 80, 3
    rows = _list(nx, ny, 20000)
    vals = np.random.default_rng(6).standard_normal((steps, 2, len(rows)))
    eps = np.random.default_rng(4).uniform(1.0, 9.0, (2, 9, 8))
    eps = np.concatenate([eps, np.ones((nb - 2, 9, 8))])
    out = _run(_problem(nx, ny, nb, rows, vals, "fp64", steps), eps, np.ones(nb))
    few = _run(_problem(nx, ny, 2, rows, vals, "fp64", steps), eps[:2], np.ones(2))
    assert np.abs(out[8]).max() > 0
    for k, (a, b) in enumerate(zip(out, few)):
        assert np.array_equal(a, b), k


@pytest.mark.parametrize("name,n", [("sheet", 5000), ("doubles", 400)])
def test_long_lists_cost_about_what_short_ones_do(name, n):
    import torch
    nx, ny, steps = 300, 243, 60
    vals = np.ones((steps, 2, n))
    if name == "sheet":
        rows = [(2, 1, 60 * ny + q) for q in range(n)]
    else:
        rows = [(c, 1, 60 * ny + q) for c in (2, 4) for q in range(n // 2)]
    eps = np.ones((1, 9, 8))
    probs = {k: _problem(nx, ny, 1, rows[:k], vals[:, :, :k], "fp64", steps, keep_history=True)
             for k in (13, n)}
    took = {k: [] for k in probs}
    for _ in range(6):
        for k, prob in probs.items():
            ev = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            prob.forward(eps)
            ev[0].record()
            prob.forward(eps)
            prob.backward()
            ev[1].record()
            torch.cuda.synchronize()
            took[k].append(ev[0].elapsed_time(ev[1]))
    assert min(took[n]) < 3 * min(took[13]), took
