"""Performance cases of the FDTD engine, measured through its public API.

A case is a dict of plain values.  ``listed()`` gives the fixed cases,
``draw(rng)`` one more of the same ranges, ``prepare(case, seed)`` what a
program holds before the call (scene on the GPU, initial fields from the
seed), ``run(state)`` one pass and its outputs, ``work(case)`` the bytes and
operations a pass cannot do without, and ``exact(case, seed)`` the outputs of
``run`` on a fresh state from a plain FP64 torch statement of the same
difference equations.

Three kinds of case:

* ``grid``: one simulation (``FDTD``, ``TMzFDTD``, ``TEzFDTD``) advanced by
  ``steps`` time steps with ``step()`` (one step) or ``step_until_n()``;
  outputs: every active field component.
* ``batch``: several grids of different sizes advanced together for one
  chunk of steps, as the job server does between two admissions; outputs:
  every active field component of every grid.
* ``design``: value and gradient of a monitor objective with respect to a
  permittivity region, for a batch of designs (forward and time-reversed
  sweep); outputs: objective, gradient.
"""

import math

import torch

import gmes_gb300 as G

COMPS = ("ex", "ey", "ez", "hx", "hy", "hz")
ACTIVE = {"3d": (0, 1, 2, 3, 4, 5), "tmz": (2, 3, 4), "tez": (0, 1, 5)}
CLASSES = {"3d": G.FDTD, "tmz": G.TMzFDTD, "tez": G.TEzFDTD}
RES = 20


def grid(name, mode, n, precision, steps, medium="dielectric", pml="cpml", cells=10, objects=8,
         bloch=False, tfsf=False):
    c = dict(kind="grid", mode=mode, nx=n[0], ny=n[1], nz=n[2] if mode == "3d" else 1,
             precision=precision, steps=steps, medium=medium, pml=pml, cells=cells,
             objects=objects, bloch=bloch, tfsf=tfsf)
    return dict(c, name=name) if name else c


def listed():
    return [
        # the 2-D example of the documentation: vacuum, 20-cell CPML, to t = 10
        grid("air2d_fp64", "tmz", (200, 200), "fp64", 286, cells=20, objects=0),
        # a user's own loop: one step() call at a time on a small 3-D grid
        grid("step_call_fp64", "3d", (48, 40, 44), "fp64", 1, cells=8),
        # a large 2-D run with a dispersive inclusion (serving mix: 2-D up to 1024^2)
        grid("tez_drude_fp64", "tez", (1000, 777), "fp64", 64, medium="drude", cells=12,
             objects=3),
        # the 3-D dielectric + CPML benchmark scene, in each arithmetic
        grid("cube256_fp64", "3d", (256, 256, 256), "fp64", 20, objects=24),
        grid("cube256_fp32", "3d", (256, 256, 256), "fp32", 20, objects=24),
        grid("ragged_df64", "3d", (181, 230, 203), "df64", 20, objects=16),
        # the 3-D dispersive + UPML + plane-wave benchmark scene
        grid("dispersive192_fp64", "3d", (192, 192, 192), "fp64", 16, medium="mixed",
             pml="upml", cells=12, objects=16, tfsf=True),
        # the same media on an odd grid in single precision, point source
        grid("dispersive_ragged_fp32", "3d", (171, 130, 149), "fp32", 24, medium="mixed",
             pml="upml", cells=12, objects=9),
        # unit cell of a photonic crystal with Bloch-periodic complex fields
        grid("bloch_cell_fp64", "3d", (64, 64, 48), "fp64", 64, pml="none", cells=0, objects=2,
             bloch=True),
        # one chunk of the serving mix: 2-D and 3-D grids advanced together
        dict(kind="batch", name="serving_mix_fp64", precision="fp64", jobs=8, steps=64, lo2=128,
             hi2=1024, lo3=64, hi3=160),
        # permittivity gradients of a batch of designs, recorded history
        dict(kind="design", name="gradients512_fp32", precision="fp32", nx=512, ny=512,
             px=64, py=64, batch=64, steps=400, cells=20, history=True),
        # the same in double precision on an odd lattice, with sqrt(N) checkpoints
        dict(kind="design", name="gradients_ckpt_fp64", precision="fp64", nx=300, ny=243, px=40,
             py=33, batch=6, steps=200, cells=16, history=False),
    ]


def _spread(rng, lo, hi):
    """An integer between lo and hi, evenly spread over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["2d", "2d", "3d", "3d", "3d", "dispersive", "bloch", "batch", "design"])
    precision = rng.choice(["fp64", "fp64", "fp32", "df64"])
    if kind == "2d":
        n = (_spread(rng, 60, 1400), _spread(rng, 60, 1400))
        medium = rng.choice(["dielectric", "dielectric", "drude", "lorentz"])
        return grid(None, rng.choice(["tmz", "tez"]), n, precision, rng.randint(40, 290),
                    medium=medium, cells=rng.randint(8, 20), objects=rng.randint(1, 6))
    if kind == "3d":
        n = [_spread(rng, 32, 260) for _ in range(3)]
        steps = 1 if rng.random() < 0.2 else rng.randint(8, 20)
        return grid(None, "3d", n, precision, steps, cells=rng.randint(6, 10),
                    objects=rng.randint(4, 24))
    if kind == "dispersive":
        n = [_spread(rng, 48, 190) for _ in range(3)]
        return grid(None, "3d", n, precision, rng.randint(8, 24),
                    medium=rng.choice(["mixed", "drude", "lorentz"]),
                    pml=rng.choice(["upml", "cpml"]), cells=rng.randint(8, 12),
                    objects=rng.randint(2, 16), tfsf=rng.random() < 0.25)
    if kind == "bloch":
        mode = rng.choice(["tmz", "tez", "3d"])
        n = [_spread(rng, 24, 96) for _ in range(3)]
        return grid(None, mode, n, "fp64", rng.randint(16, 128), pml="none", cells=0,
                    objects=rng.randint(1, 4), bloch=True)
    if kind == "batch":
        return dict(kind="batch", precision=rng.choice(["fp64", "fp32"]),
                    jobs=rng.randint(3, 10), steps=rng.randint(16, 64), lo2=128,
                    hi2=_spread(rng, 256, 1024), lo3=40, hi3=_spread(rng, 64, 150))
    nx, ny = _spread(rng, 120, 512), _spread(rng, 120, 512)
    return dict(kind="design", precision=rng.choice(["fp32", "fp32", "fp64"]), nx=nx, ny=ny,
                px=rng.randint(8, nx // 5), py=rng.randint(8, ny // 5),
                batch=_spread(rng, 1, 24), steps=rng.randint(60, 300),
                cells=rng.randint(10, 20), history=rng.random() < 0.6)


# ---------------------------------------------------------------------------
# Scenes.  A scene is plain data (sizes, shapes, media, source, initial wave
# packets), made from the seed; _simulation() hands it to the framework and
# _Exact steps it in plain torch.
# ---------------------------------------------------------------------------
def _uniform(rng, lo, hi):
    return lo + (hi - lo) * torch.rand((), generator=rng, dtype=torch.float64).item()


def _medium(kind, rng):
    """(model, eps_inf, Drude or Lorentz poles, critical points)."""
    if kind == "drude":
        return ("drude", 1.0, ((9.0, 0.07),), ())
    if kind == "lorentz":
        return ("lorentz", 1.0, ((2.0, 3.0, 0.1),), ())
    if kind == "dcp":
        cps = tuple((_uniform(rng, 0.5, 2.0), _uniform(rng, -1.5, 1.5), _uniform(rng, 2.0, 5.0),
                     _uniform(rng, 0.2, 1.0)) for _ in range(2))
        return ("dcp", 1.1, ((7.0, 0.2),), cps)
    return ("dielectric", _uniform(rng, 1.0, 12.0), (), ())


def _scene(case, seed):
    rng = torch.Generator().manual_seed(int(seed))
    mode = case["mode"]
    dims = 3 if mode == "3d" else 2
    n = (case["nx"], case["ny"], case["nz"])
    dx = 1.0 / RES
    inner = [n[a] * dx / 2 - (case["cells"] + 1) * dx for a in range(dims)]
    mixed = case["medium"] == "mixed"
    shapes = []
    for q in range(case["objects"]):
        r = _uniform(rng, 0.12, 0.35) * min(inner) * (0.6 if case["objects"] > 4 else 1.0)
        center = [_uniform(rng, r - h, h - r) for h in inner] + [0.0] * (3 - dims)
        kind = case["medium"]
        if mixed:
            kind = "lorentz" if q == 0 else "dcp" if q == 1 else "drude"
        sphere = _uniform(rng, 0.0, 1.0) < 0.5 or (mixed and q > 0)
        half = [r, r, r]
        if mixed and q == 0:  # the slab of the dispersive scene
            sphere, center = False, [0.0, 0.0, 0.35 * inner[2]]
            half = [0.97 * inner[0], 0.97 * inner[1], 0.08 * inner[2]]
        shapes.append(("sphere" if sphere else "block", center, half, _medium(kind, rng)))
    packets = []
    for _ in range(3):
        packets.append(dict(
            center=[_uniform(rng, -0.6, 0.6) * h for h in inner] + [0.0] * (3 - dims),
            k=[_uniform(rng, -6.0, 6.0) for _ in range(dims)] + [0.0] * (3 - dims),
            width=0.3 * min(inner) + 2 * dx, phase=_uniform(rng, 0.0, 2 * math.pi),
            amp=[_uniform(rng, -1.0, 1.0) for _ in range(6)]))
    dispersive = case["medium"] != "dielectric"
    src_comp = 2 if mode != "tez" else 0
    src = dict(comp=src_comp, idx=[int(n[a] * 0.4) for a in range(dims)] + [0] * (3 - dims),
               freq=0.8 + 0.2 * _uniform(rng, 0.0, 1.0))
    return dict(
        mode=mode, n=n, dx=dx, dims=dims, shapes=shapes, packets=packets, src=src,
        background=2.25 if mixed else 1.0, ratio=0.6 if dispersive else 0.99,
        pml=case["pml"], thickness=case["cells"] * dx,
        bloch=tuple(_uniform(rng, -1.0, 1.0) if a < dims else 0.0 for a in range(3))
        if case["bloch"] else None, tfsf=case["tfsf"], precision=case["precision"])


def _offset(c, a):
    """Yee offset of component c along axis a, in cells."""
    if c < 3:
        return 0.5 if a == c else 0.0
    return 0.0 if a == c - 3 else -0.5


def _shape(scene, c):
    n = scene["n"]
    return tuple(n[a] if a == c % 3 else n[a] + 1 for a in range(3))


def _axes(scene, c, shape, device, first=(0, 0, 0)):
    """Coordinates of component c along the three axes, broadcastable."""
    out = []
    for a in range(3):
        v = (torch.arange(shape[a], device=device, dtype=torch.float64) + (first[a]
             + _offset(c, a))) * scene["dx"] - 0.5 * scene["n"][a] * scene["dx"]
        out.append(v.view([-1 if b == a else 1 for b in range(3)]))
    return out


def _packet_field(scene, c, shape, device):
    """Initial value of component c: three windowed wave packets."""
    x = _axes(scene, c, shape, device)
    f = torch.zeros(shape, dtype=torch.float64, device=device)
    for p in scene["packets"]:
        r2 = sum((x[a] - p["center"][a]) ** 2 for a in range(scene["dims"]))
        phase = sum(p["k"][a] * x[a] for a in range(scene["dims"])) + p["phase"]
        f += p["amp"][c] * torch.exp(-r2 / (2 * p["width"] ** 2)) * torch.cos(phase)
    return f


def _material(medium):
    model, eps, poles, cps = medium
    if model == "drude":
        return G.Drude(eps_inf=eps, dps=[G.DrudePole(omega=w, gamma=g) for w, g in poles])
    if model == "lorentz":
        return G.Lorentz(eps_inf=eps, lps=[G.LorentzPole(amp=a, omega=w, gamma=g)
                                           for a, w, g in poles])
    if model == "dcp":
        return G.DcpAde(eps_inf=eps, dps=[G.DrudePole(omega=w, gamma=g) for w, g in poles],
                        cps=[G.CriticalPoint(amp=a, phi=p, omega=w, gamma=g)
                             for a, p, w, g in cps])
    return G.Dielectric(eps_inf=eps)


def _simulation(scene):
    n, dx, dims = scene["n"], scene["dx"], scene["dims"]
    size = [n[a] * dx if a < dims else 0 for a in range(3)]
    geom = [G.DefaultMedium(material=G.Dielectric(eps_inf=scene["background"]))]
    for kind, center, half, medium in scene["shapes"]:
        if kind == "sphere":
            geom.append(G.Sphere(material=_material(medium), center=center, radius=half[0]))
        else:
            geom.append(G.Block(material=_material(medium), center=center,
                                size=[2 * h for h in half]))
    if scene["pml"] != "none":
        pml = G.Cpml() if scene["pml"] == "cpml" else G.Upml()
        geom.append(G.Shell(material=pml, thickness=scene["thickness"]))
    s = scene["src"]
    if scene["tfsf"]:
        box = [0.9 * (v - 2 * scene["thickness"]) for v in size]
        src = G.TotalFieldScatteredField(src_time=G.Continuous(freq=s["freq"], width=2.0),
                                         center=(0, 0, 0), size=box, direction=(0, 0, 1),
                                         polarization=(1, 0, 0))
    else:
        at = [(s["idx"][a] + _offset(s["comp"], a)) * dx - 0.5 * n[a] * dx for a in range(3)]
        src = G.PointSource(src_time=G.Continuous(freq=s["freq"], width=2.0), center=at,
                            component=(G.Jx, G.Jy, G.Jz)[s["comp"]])
    sim = CLASSES[scene["mode"]](G.Cartesian(size=size, resolution=RES), geom, [src],
                                 courant_ratio=scene["ratio"], bloch=scene["bloch"],
                                 verbose=False, precision=scene["precision"])
    sim.init()
    # a run that is under way: wave packets on the grid, the source still rising
    for c in ACTIVE[scene["mode"]]:
        if c < 3:
            f = _packet_field(scene, c, _shape(scene, c), "cuda")
            if scene["bloch"] is not None:
                f = (f * (1 + 0.5j)).cpu().numpy()
            getattr(sim, COMPS[c])[:] = f
    return sim


def _fields(sim, mode):
    """The active components: single precision as stored, the others as FP64."""
    if sim.precision == "fp32":
        return {COMPS[c]: sim.engine.tensor(c) for c in ACTIVE[mode]}
    return {COMPS[c]: getattr(sim, COMPS[c]).tensor() for c in ACTIVE[mode]}


def _batch_cases(case, seed):
    """The grids of a batch: even ones 2-D TMz, odd ones 3-D, media in turn; sizes
    spread over the range (the same for every seed)."""
    out = []
    m = max(1, (case["jobs"] + 1) // 2 - 1)
    for q in range(case["jobs"]):
        t = (q // 2) / m
        kind = ("dielectric", "drude", "lorentz")[q % 3]
        if q % 2 == 0:
            side = int(case["lo2"] + (case["hi2"] - case["lo2"]) * t)
            g = grid(None, "tmz", (side, side), case["precision"], case["steps"], medium=kind,
                     cells=8 + q, objects=1)
        else:
            side = int(case["lo3"] + (case["hi3"] - case["lo3"]) * t * t)
            g = grid(None, "3d", (side, side, side), case["precision"], case["steps"],
                     medium=kind, cells=8 + q % 8, objects=1)
        out.append(g)
    return out


def _design_parts(case, seed):
    """(space, geometry, sources, design, monitor, eps) of a differentiation problem."""
    from gmes_gb300.adjoint import DesignRegion
    dx = 1.0 / RES
    nx, ny, pml = case["nx"], case["ny"], case["cells"]
    geom = [G.DefaultMedium(material=G.Dielectric()),
            G.Shell(material=G.Cpml(), thickness=pml * dx)]
    i_src, js = _design_source(case)
    src = [G.PointSource(src_time=G.Continuous(freq=1.0, width=2.0),
                         center=(i_src * dx - nx * dx / 2, j * dx - ny * dx / 2, 0),
                         component=G.Jz) for j in js]
    space = G.Cartesian(size=(nx * dx, ny * dx, 0), resolution=RES)
    (d0, dn), (m0, mn) = _design_boxes(case)

    def region(lo, n):
        return DesignRegion(center=[(lo[a] + n[a] / 2) * dx - (nx, ny)[a] * dx / 2
                                    for a in range(2)], size=[n[a] * dx for a in range(2)])

    rng = torch.Generator().manual_seed(int(seed))
    eps = 1.0 + 11.0 * torch.rand((case["batch"], *dn), generator=rng, dtype=torch.float64)
    return space, geom, src, region(d0, dn), region(m0, mn), eps


def _design_boxes(case):
    """((lo, n) of the design region, (lo, n) of the monitor), in Ez lattice points."""
    nx, ny, px, py = case["nx"], case["ny"], case["px"], case["py"]
    return (((nx - px) // 2, (ny - py) // 2), (px, py)), (((nx + px) // 2 + 4, ny // 2 - 4), (8, 8))


def _design_source(case):
    return (case["nx"] - case["px"]) // 2 - 6, range(case["cells"] + 1, case["ny"] - case["cells"])


def prepare(case, seed):
    if case["kind"] == "grid":
        return dict(case=case, sim=_simulation(_scene(case, seed)))
    if case["kind"] == "batch":
        from gmes_gb300.batch import Batch
        cases = _batch_cases(case, seed)
        sims = [_simulation(_scene(c, seed + 1000 * q)) for q, c in enumerate(cases)]
        return dict(case=case, sims=sims, modes=[c["mode"] for c in cases], done=0,
                    batch=Batch([s.engine for s in sims]))
    from gmes_gb300.adjoint import TMzAdjoint
    space, geom, src, design, monitor, eps = _design_parts(case, seed)
    problem = TMzAdjoint(space, geom, src, design, monitor, case["steps"], batch=case["batch"],
                         precision=case["precision"], keep_history=case["history"])
    return dict(case=case, problem=problem, eps=eps.cuda())


def run(state):
    case = state["case"]
    if case["kind"] == "grid":
        sim = state["sim"]
        if case["steps"] == 1:
            sim.step()
        else:
            sim.step_until_n(sim.time_step.n + case["steps"])
        return _fields(sim, case["mode"])
    if case["kind"] == "batch":
        b, k = state["batch"], case["steps"]
        b.run([k] * len(state["sims"]), [float(state["done"])] * len(state["sims"]))
        b.synchronize()
        state["done"] += k
        return [_fields(s, m) for s, m in zip(state["sims"], state["modes"])]
    eps = state["eps"].detach().requires_grad_(True)
    value = state["problem"].objective(eps)
    value.sum().backward()
    return {"value": value.detach(), "gradient": eps.grad}


# ---------------------------------------------------------------------------
# Work.  Per time step every active field value is read once and written
# once, every active point's one-byte material id is read, and the state of
# the absorbing layer and of dispersive points is read and written.  A curl
# update of one component takes 8 operations (four differences and multiply-
# adds); the state terms are counted the same way.
# ---------------------------------------------------------------------------
def _grid_work(case):
    n = (case["nx"], case["ny"], case["nz"])
    dims = 3 if case["mode"] == "3d" else 2
    cells = float(n[0] * n[1] * n[2])
    ncomp = len(ACTIVE[case["mode"]])
    es = 4 if case["precision"] == "fp32" else 16 if case["bloch"] else 8
    nbytes, flops = ncomp * cells * (2 * es + 1), ncomp * cells * 8 * (2 if case["bloch"] else 1)
    if case["pml"] != "none":
        for a in range(dims):
            slab = cells * min(1.0, 2 * case["cells"] / n[a])
            # CPML: one psi of the components whose curl crosses the axis
            per = (4 if dims == 3 else 2) if case["pml"] == "cpml" else ncomp / dims
            nbytes += slab * per * 2 * es
            flops += slab * per * 6
    if case["medium"] != "dielectric" and case["objects"]:
        # inclusions fill a few per cent of the grid; two state values per pole
        nbytes += 0.03 * cells * (ncomp / 2) * 4 * es
        flops += 0.03 * cells * (ncomp / 2) * 12
    return nbytes * case["steps"], flops * case["steps"]


def work(case):
    if case["kind"] == "grid":
        b, f = _grid_work(case)
    elif case["kind"] == "batch":
        parts = [_grid_work(c) for c in _batch_cases(case, 0)]
        b, f = sum(p[0] for p in parts), sum(p[1] for p in parts)
    else:
        # forward and adjoint sweep: three fields read and written per step
        es = 4 if case["precision"] == "fp32" else 8
        points = float(case["nx"] * case["ny"] * case["batch"] * case["steps"])
        b = points * 2 * 6 * es + 2 * case["px"] * case["py"] * case["batch"] * case["steps"] * es
        f = points * (24 + 32)
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------------------------
# Exact: the same difference equations in FP64 torch, over whole arrays on the
# periodic lattice of cells.  E_c of cell (i, j, k) sits at the component's
# array index (i, j, k); H_c of the cell at that index plus one along its two
# transverse axes.  The layers' profiles and the poles' coefficients follow
# the published forms (Taflove & Hagness; Roden & Gedney; Gedney; Vial).
# ---------------------------------------------------------------------------
def _profile(scene, c, a, dt, device):
    """Layer coefficients of component c along axis a, one row per cell."""
    n, dx = scene["n"][a], scene["dx"]
    first = 1 if c >= 3 and a != c - 3 else 0
    w = (torch.arange(n, device=device, dtype=torch.float64) + first + _offset(c, a)) * dx \
        - 0.5 * n * dx
    d, h = scene["thickness"], 0.5 * n * dx
    cpml = scene["pml"] == "cpml"
    m, kmax, ratio = (3.4, 1.0, 0.65) if cpml else (3.6, 4.6, 0.745)
    inside = (h - w.abs()) <= d
    if a >= scene["dims"] or scene["pml"] == "none":
        inside = torch.zeros_like(inside)
    depth = torch.where(inside, ((h - w.abs()) / d if d else w * 0).clamp(0, 1),
                        torch.ones_like(w))
    sigma = ratio * 0.8 * (m + 1) / dx * (1 - depth) ** m
    kappa = 1 + (kmax - 1) * (1 - depth) ** m
    if cpml or scene["pml"] == "none":
        alpha = torch.where(inside, 0.8 * depth ** 4.8, torch.zeros_like(w))
        b = torch.exp(-(sigma / kappa + alpha) * dt)
        den = (sigma + kappa * alpha) * kappa
        cc = torch.where(den > 0, sigma * (b - 1) / torch.where(den > 0, den, den + 1), den * 0)
        rows = (b, cc / dx, 1 / (kappa * dx))
    else:
        rows = ((2 * kappa - sigma * dt) / (2 * kappa + sigma * dt),
                2 * dt / (2 * kappa + sigma * dt), 1 / (2 * kappa + sigma * dt),
                2 * kappa + sigma * dt, 2 * kappa - sigma * dt)
    return [r.view([-1 if b == a else 1 for b in range(3)]) for r in rows]


def _source_value(freq, t, width=2.0):
    """Continuous source with a Hann-window start (complex amplitude)."""
    env = math.sin(0.5 * math.pi * t / width) ** 2 if t < width else 1.0
    ph = 2 * math.pi * freq * t
    return env * complex(math.cos(ph), math.sin(ph))


class _Exact:
    def __init__(self, scene):
        self.s = scene
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.act = ACTIVE[scene["mode"]]
        self.dt = scene["ratio"] * math.sqrt(scene["background"]) * scene["dx"] \
            / math.sqrt(scene["dims"])
        self.cx = scene["bloch"] is not None
        n, dev = scene["n"], self.dev
        kind = torch.complex128 if self.cx else torch.float64
        self.f, self.last = {}, {}
        self.psi = {}
        for c in range(6):
            self.f[c] = torch.zeros(n, dtype=kind, device=dev)
            if c in self.act and c < 3:
                v = _packet_field(scene, c, n, dev)
                self.f[c] = v * (1 + 0.5j) if self.cx else v
        self.eps, self.masks = {}, {c: [] for c in range(6)}
        for c in self.act:
            x = _axes(scene, c, n, dev)
            eps = torch.full(n, scene["background"] if c < 3 else 1.0, dtype=torch.float64,
                             device=dev)
            owner = torch.full(n, -1, dtype=torch.int16, device=dev)
            if c < 3:
                for q, (shape, center, half, medium) in enumerate(scene["shapes"]):
                    r = [x[a] - center[a] for a in range(3)]
                    if shape == "sphere":
                        m = torch.sqrt(r[0] ** 2 + r[1] ** 2 + r[2] ** 2) <= half[0]
                    else:
                        m = (r[0].abs() <= half[0]) & (r[1].abs() <= half[1]) \
                            & (r[2].abs() <= half[2])
                    owner[m.expand(n)] = q
                for q, (_, _, _, medium) in enumerate(scene["shapes"]):
                    eps[owner == q] = medium[1]
                for q, (_, _, _, medium) in enumerate(scene["shapes"]):
                    if medium[0] != "dielectric":
                        at = (owner == q).nonzero(as_tuple=True)
                        self.masks[c].append((at, *self._poles(medium, at[0].numel(), kind)))
            self.eps[c] = eps
            rows = [_profile(scene, c, a, self.dt, dev) for a in range(3)]
            zero = torch.zeros(n, dtype=kind, device=dev)
            self.psi[c] = [rows, zero.clone(), zero.clone()]

    def _poles(self, medium, count, kind):
        """Coefficient rows and state of the poles of one inclusion."""
        model, eps, poles, cps = medium
        dt = self.dt
        z = lambda: torch.zeros(count, dtype=kind, device=self.dev)  # noqa: E731
        if model in ("drude", "lorentz"):
            rows = []
            for p in poles:
                amp, w, g = (1.0, *p) if model == "drude" else p
                den = dt * g + 2
                stiff = 0.0 if model == "drude" else 2 * (dt * w) ** 2
                rows.append([(dt * g - 2) / den, (4 - stiff) / den, 2 * amp * (dt * w) ** 2 / den,
                             z(), z()])
            return model, rows, [], (dt / eps, -1 / eps, 1.0), None
        rows, crit = [], []
        for w, g in poles:
            den = dt * g + 2
            rows.append([(dt * g - 2) / den, 4 / den, 0.5 * (dt * w) ** 2 / den, z(), z()])
        for amp, phi, w, g in cps:
            den = (dt * g + 2) ** 2 + (dt * w) ** 2
            sp, cp = math.sin(phi), math.cos(phi)
            crit.append([-((dt * g - 2) ** 2 + (dt * w) ** 2) / den,
                         2 * (4 - dt ** 2 * (g ** 2 + w ** 2)) / den,
                         2 * dt * amp * w * (dt * cp * w + sp * (2 - dt * g)) / den,
                         4 * dt ** 2 * amp * w * (cp * w - sp * g) / den,
                         2 * dt * amp * w * (dt * cp * w - sp * (2 + dt * g)) / den, z(), z()])
        sa = sum(r[2] for r in rows)
        s2, s3, s4 = (sum(r[k] for r in crit) for k in (2, 3, 4))
        den = sa + s4 + eps
        return model, rows, crit, (dt / den, 1 / den, -(sa + s2) / den,
                                   -(2 * sa + s3 - eps) / den), z()

    def _shift(self, f, a, step):
        """f at the next (step +1) or previous (-1) cell along a, Bloch-periodic."""
        out = torch.roll(f, -step, a)
        if self.cx and self.s["bloch"][a] != 0.0:
            n = self.s["n"][a]
            kl = self.s["bloch"][a] * n * self.s["dx"] * step
            out.narrow(a, n - 1 if step > 0 else 0, 1).mul_(complex(math.cos(kl), math.sin(kl)))
        return out

    def _update(self, c):
        a1, a2 = (c + 1) % 3, (c + 2) % 3
        e = c < 3
        p, q = (3 + a2, 3 + a1) if e else (a2, a1)
        zero = torch.zeros((), dtype=self.f[c].dtype, device=self.dev)
        sgn = -1 if e else 1
        d1 = (self._shift(self.f[p], a1, sgn) - self.f[p]) * sgn if p in self.act else zero
        d2 = (self._shift(self.f[q], a2, sgn) - self.f[q]) * sgn if q in self.act else zero
        f, dx = self.f[c], self.s["dx"]
        rows, s1, s2 = self.psi[c]
        curl = None
        old = [f[m[0]].clone() for m in self.masks[c]]
        if self.masks[c]:
            curl = ((d1 - d2) / dx)
        if self.s["pml"] == "upml":
            own = c % 3
            x = (d1 - d2) / dx
            new = rows[a1][0] * s1 + rows[a1][1] * (x if e else -x)
            f = rows[a2][0] * f + rows[a2][2] * (rows[own][3] * new - rows[own][4] * s1) \
                / self.eps[c]
            s1.copy_(new)
        else:
            s1.mul_(rows[a1][0]).add_(rows[a1][1] * d1)
            s2.mul_(rows[a2][0]).add_(rows[a2][1] * d2)
            x = s1 - s2 + rows[a1][2] * d1 - rows[a2][2] * d2
            f = f + self.dt / self.eps[c] * (x if e else -x)
        for m, now in zip(self.masks[c], old):
            f[m[0]] = self._dispersive(m, now, curl[m[0]])
        self.f[c] = f

    @staticmethod
    def _dispersive(m, now, curl):
        _, model, rows, crit, k, e_old = m
        if model != "dcp":
            total = 0
            for r in rows:
                new = r[0] * r[3] + r[1] * r[4] + r[2] * now
                total = total + (new - r[4])
                r[3], r[4] = r[4], new
            return k[0] * curl + k[1] * total + k[2] * now
        acc = sum((1 - r[1]) * r[4] - r[0] * r[3] for r in rows)
        acc = acc + sum((1 - r[1]) * r[6] - r[0] * r[5] for r in crit)
        new = k[0] * curl + k[1] * acc + k[2] * e_old + k[3] * now
        for r in rows:
            r[3], r[4] = r[4], r[0] * r[3] + r[1] * r[4] + r[2] * (e_old + 2 * now + new)
        for r in crit:
            r[5], r[6] = r[6], (r[0] * r[5] + r[1] * r[6] + r[2] * e_old + r[3] * now
                                + r[4] * new)
        e_old.copy_(now)
        return new

    def step(self, n):
        self.last = {c: self.f[c] for c in self.act if c >= 3}
        for c in self.act:
            if c < 3:
                self._update(c)
        s = self.s["src"]
        at = tuple(s["idx"])
        v = _source_value(s["freq"], self.dt * (n + 0.5))
        c = s["comp"]
        self.f[c][at] -= self.dt * (v if self.cx else v.real) / self.eps[c][at]
        for c in self.act:
            if c >= 3:
                self._update(c)

    def outputs(self):
        """The component arrays with their ghost planes: E's copied from the
        present values, H's from those before the last step."""
        out = {}
        for c in self.act:
            f = self.f[c] if c < 3 else self.last[c]
            for a in ((c + 1) % 3, (c + 2) % 3):
                if c < 3:
                    g = self._shift(f, a, 1).narrow(a, f.shape[a] - 1, 1)
                    f = torch.cat((f, g), a)
                else:
                    g = self._shift(f, a, -1).narrow(a, 0, 1)
                    f = torch.cat((g, f), a)
            if c >= 3:
                sl = [slice(None)] * 3
                for a in ((c + 1) % 3, (c + 2) % 3):
                    sl[a] = slice(1, None)
                f[tuple(sl)] = self.f[c]
            out[COMPS[c]] = f
        return out


def _exact_grid(case, seed):
    if case["tfsf"]:
        return None
    x = _Exact(_scene(case, seed))
    for n in range(case["steps"]):
        x.step(n)
    return x.outputs()


def _exact_design(case, seed):
    """Objective and gradient by reverse mode over segments of the TMz steps."""
    from torch.utils.checkpoint import checkpoint
    points = case["nx"] * case["ny"] * case["batch"]
    if points * case["steps"] > 1.2e10 or not torch.cuda.is_available():
        return None
    dev, dx, nsteps = "cuda", 1.0 / RES, case["steps"]
    n = (case["nx"], case["ny"], 1)
    scene = dict(n=n, dx=dx, dims=2, pml="cpml", thickness=case["cells"] * dx)
    dt = 0.99 * dx / math.sqrt(2)
    rng = torch.Generator().manual_seed(int(seed))
    (d0, dn), (m0, mn) = _design_boxes(case)
    eps = 1.0 + 11.0 * torch.rand((case["batch"], *dn), generator=rng, dtype=torch.float64)
    eps = eps.to(dev).requires_grad_(True)
    rows = {}
    for c, a in ((2, 0), (2, 1), (3, 1), (4, 0)):
        rows[c, a] = [r.reshape((-1, 1) if a == 0 else (1, -1))
                      for r in _profile(scene, c, a, dt, dev)]
    i_src, js = _design_source(case)
    line = torch.zeros(n[:2], dtype=torch.float64, device=dev)
    line[i_src, js.start:js.stop] = dt

    def segment(first, count, eps, e, hx, hy, p1, p2, px, py, value):
        pad = (d0[1], n[1] - d0[1] - dn[1], d0[0], n[0] - d0[0] - dn[0])
        cdt = dt / torch.nn.functional.pad(eps - 1, pad).add(1)
        for s in range(first, first + count):
            a, b = hy - torch.roll(hy, 1, 1), hx - torch.roll(hx, 1, 2)
            p1 = rows[2, 0][0] * p1 + rows[2, 0][1] * a
            p2 = rows[2, 1][0] * p2 + rows[2, 1][1] * b
            e = e + cdt * (p1 - p2 + rows[2, 0][2] * a - rows[2, 1][2] * b) \
                - line * _source_value(1.0, dt * (s + 0.5)).real
            a, b = torch.roll(e, -1, 2) - e, torch.roll(e, -1, 1) - e
            px = rows[3, 1][0] * px + rows[3, 1][1] * a
            py = rows[4, 0][0] * py + rows[4, 0][1] * b
            hx = hx - dt * (px + rows[3, 1][2] * a)
            hy = hy + dt * (py + rows[4, 0][2] * b)
            m = e[:, m0[0]:m0[0] + mn[0], m0[1]:m0[1] + mn[1]]
            value = value + dt * (m * m).sum((1, 2))
        return e, hx, hy, p1, p2, px, py, value

    state = [torch.zeros((case["batch"], *n[:2]), dtype=torch.float64, device=dev)
             for _ in range(7)] + [torch.zeros(case["batch"], dtype=torch.float64, device=dev)]
    k = max(1, int(math.sqrt(nsteps) / 2))
    for first in range(0, nsteps, k):
        state = checkpoint(segment, first, min(k, nsteps - first), eps, *state,
                           use_reentrant=False)
    state[-1].sum().backward()
    return {"value": state[-1].detach(), "gradient": eps.grad}


def exact(case, seed):
    if case["kind"] == "grid":
        return _exact_grid(case, seed)
    if case["kind"] == "batch":
        return [_exact_grid(c, seed + 1000 * q) for q, c in enumerate(_batch_cases(case, seed))]
    return _exact_design(case, seed)
