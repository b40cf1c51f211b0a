"""A small grid's chunk of steps in one launch against the same steps as
half-step launches.

``gmes_step`` advances small and 2-D grids with one cooperative kernel;
``gmes_half_step`` always launches the ghost copy, cell update and source
kernels.  Both run the same arithmetic on every point, so the whole arrays,
ghost planes included, must agree bit for bit: 1, 2 and more steps, cell
counts that are no multiple of a warp, every mask of active components,
sources on the domain's edge, classes and layers beyond the shared-memory
tables, complex fields, and chunks of different lengths one after another.
"""
import numpy as np
import pytest

import gmes_gb300 as G

pytestmark = pytest.mark.gpu


def _scene(cls, size, res, precision, medium="dielectric", pml="cpml", bloch=None, many=False,
           edge=False, kappa=1.0, comp=None):
    size = tuple(size)
    live = [a for a in range(3) if size[a] > 0]
    rng = np.random.default_rng(7)
    geom = [G.DefaultMedium(material=G.Dielectric())]
    half = [0.5 * v for v in size]
    small = min(half[a] for a in live)
    mats = {"dielectric": G.Dielectric(eps_inf=3.0),
            "drude": G.Drude(eps_inf=1, dps=(G.DrudePole(omega=9.0, gamma=0.07),)),
            "dcp": G.DcpAde(eps_inf=1.1, dps=(G.DrudePole(omega=7.0, gamma=0.2),),
                            cps=(G.CriticalPoint(amp=1.0, phi=0.4, omega=3.0, gamma=0.4),))}
    geom.append(G.Sphere(material=mats[medium], center=(0, 0, 0), radius=0.4 * small))
    if many:  # more classes than the shared-memory table holds
        for q in range(40):
            c = [0.5 * half[a] * rng.uniform(-1, 1) if a in live else 0.0 for a in range(3)]
            geom.append(G.Sphere(material=G.Dielectric(eps_inf=1.5 + 0.1 * q), center=c,
                                 radius=0.15 * small))
    d = 0.25 * small
    if pml == "cpml":
        geom.append(G.Shell(material=G.Cpml(kappa_max=kappa), thickness=d))
    elif pml == "upml":
        geom.append(G.Shell(material=G.Upml(), thickness=d))
    elif pml == "two":  # a second layer, beyond the tables
        geom.append(G.Shell(material=G.Cpml(), thickness=d))
        geom.append(G.Shell(material=G.Cpml(m=3.0), thickness=0.5 * d))
    src = [G.PointSource(src_time=G.Continuous(freq=0.9, width=1.0), center=(0.1, 0.05, 0.02),
                         component=comp or G.Jz)]
    if edge:  # field and current sources on the first and last planes
        at = [-half[a] if a in live else 0.0 for a in range(3)]
        src.append(G.PointSource(src_time=G.Continuous(freq=0.7, width=1.0), center=at,
                                 component=G.Ez))
        at = [half[a] - 0.5 / res if a in live else 0.0 for a in range(3)]
        src.append(G.PointSource(src_time=G.Continuous(freq=0.6, width=1.0), center=at,
                                 component=G.Hy))
    return cls(G.Cartesian(size=size, resolution=res), geom, src, courant_ratio=0.6, bloch=bloch,
               verbose=False, precision=precision)


CASES = {
    "tmz_41x37": dict(cls=G.TMzFDTD, size=(4.1, 3.7, 0), edge=True),
    "tmz_one_row": dict(cls=G.TMzFDTD, size=(0.1, 6.3, 0), pml="none"),
    "tez_33x65_drude": dict(cls=G.TEzFDTD, size=(3.3, 6.5, 0), medium="drude", comp=G.Jx),
    "tez_kappa": dict(cls=G.TEzFDTD, size=(3.3, 4.7, 0), kappa=4.0, comp=G.Jy),
    "tmx_40x31": dict(cls=G.TMxFDTD, size=(0, 4.0, 3.1), comp=G.Jx),
    "tey_29x33": dict(cls=G.TEyFDTD, size=(2.9, 0, 3.3), comp=G.Jx),
    "temz_1d": dict(cls=G.TEMzFDTD, size=(0, 0, 20.1), comp=G.Jx),
    "cube_19x21x17": dict(cls=G.FDTD, size=(1.9, 2.1, 1.7), edge=True),
    "cube_kappa": dict(cls=G.FDTD, size=(2.0, 1.8, 2.2), kappa=5.0),
    "cube_many_classes": dict(cls=G.FDTD, size=(2.4, 2.0, 2.2), many=True),
    "cube_two_layers": dict(cls=G.FDTD, size=(2.4, 2.4, 2.0), pml="two"),
    "cube_dcp_upml": dict(cls=G.FDTD, size=(2.2, 2.0, 1.9), medium="dcp", pml="upml"),
    "cube_two_rounds": dict(cls=G.FDTD, size=(5.1, 5.3, 4.8), medium="drude"),
    "tmz_wide": dict(cls=G.TMzFDTD, size=(30.1, 44.3, 0), medium="dcp"),
}
RUN = [(n, p) for n in CASES for p in ("fp64", "fp32", "df64")]
RUN += [("bloch_tez", "fp64"), ("bloch_cube", "fp64")]
CASES["bloch_tez"] = dict(cls=G.TEzFDTD, size=(2.3, 3.1, 0), bloch=(0.4, -0.3, 0), pml="none",
                          comp=G.Jx)
CASES["bloch_cube"] = dict(cls=G.FDTD, size=(1.7, 1.9, 2.1), bloch=(0.4, -0.3, 0.2),
                           medium="drude")


def _start(sim):
    sim.init()
    rng = np.random.default_rng(3)
    for comp in sim.e_field_compnt + sim.h_field_compnt:  # ghost planes too
        v = rng.standard_normal(sim.field[comp].shape)
        sim.field[comp][:] = v * (1 + 0.3j) if sim.cmplx else v
    return sim.engine


@pytest.mark.parametrize("name,precision", RUN)
def test_one_launch_equals_half_step_launches(name, precision):
    a = _start(_scene(res=10, precision=precision, **CASES[name]))
    b = _start(_scene(res=10, precision=precision, **CASES[name]))
    assert a.step_launches(7) == 1
    n = 0
    for k in (1, 2, 7):
        a.step(k, n0=float(n))
        b.stage_sources(float(n), k)
        for s in range(k):
            b.half_step(0, s)
            b.half_step(1, s)
        b.synchronize()
        a.synchronize()
        n += k
        for c in range(6):
            fa, fb = a.fields[c].cpu().numpy(), b.fields[c].cpu().numpy()
            assert np.isfinite(fa).all()
            assert np.array_equal(fa, fb), (k, c)
            if a.aux[c] is not None:
                assert np.array_equal(a.aux[c].cpu().numpy(), b.aux[c].cpu().numpy()), (k, c)


def test_route():
    """Many sources, large 3-D grids and probes keep the half-step launches."""
    sim = _scene(G.FDTD, (1.6, 1.6, 1.6), 10, "fp64")
    sim.src_list = sim.src_list + [
        G.PointSource(src_time=G.Continuous(freq=0.9), center=(0.1 * (q % 8) - 0.4, 0.1 * (q // 8)
                                                               - 0.4, 0), component=G.Jx)
        for q in range(65)]
    for s in sim.src_list:
        s.init(sim.geom_tree, sim.space, False)
    sim.init()
    assert sim.engine.step_launches(3) == 3 * 6
    sim = _scene(G.FDTD, (8.0, 8.0, 8.0), 10, "fp64")
    sim.init()
    assert sim.engine.step_launches(3) == 3 * 6
    sim = _scene(G.TMzFDTD, (4.0, 3.0, 0), 10, "fp64")
    sim.init()
    assert sim.engine.step_launches(3) == 1
    sim.engine.set_probes([(2, 5)])
    assert sim.engine.step_launches(3) == 3 * 8
