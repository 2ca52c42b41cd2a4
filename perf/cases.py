"""Performance cases of the GB300 solver: what its users have it do, through the public Python layer
(gbturbo.Solver, gbturbo.WarmStart, speedline.make_points), over the range of this repository's own
tests, generators and benchmark.

Kinds of case:
  solve   driver iterations (Solver.iterate with its history) of one or more operating points, then the
          flow field to the host: a stretch of a solve between two looks at it
  calls   the same iterations through the reference's call surface, one solver_step and one integrals
          call per iteration, as a C++ host drives the library
  train   Adam steps of the warm-start network on a set of solved fields (WarmStart.train)
  infer   the network on rows of features (WarmStart.forward)

listed() holds fixed cases, draw() further ones of the same ranges, prepare() what a program has in hand
before the call, run() one pass, work() the bytes and operations of a pass that no implementation can do
without, exact() the outputs in 64 bits where plain numpy can give them.
"""
import os
import sys
import tempfile

import numpy as np

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                    "3d-fluid-numerical-simulation-software_gb300")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import gbturbo  # noqa: E402
import meshgen  # noqa: E402
import speedline  # noqa: E402

P_TOTAL = 101325.0

#: numerical options of a variant on top of the generators' defaults (Navier-Stokes, Baldwin-Lomax,
#: Roe + MUSCL3 on primitives, local time step): the ones the tests and the benchmark run
VARIANTS = {
    "default": {},
    "sw_nnd": {"scheme": "200", "recon": "100"},            # Steger-Warming with NND
    "cons_laminar": {"recon_var": "100", "recon": "400", "turb": "0"},
    "jst": {"scheme": "100", "k2": "0.5", "k4": "32.0"},    # central scheme with artificial dissipation
    "sa": {"turb": "200"},                                  # Spalart-Allmaras (single grid only)
}

#: the benchmark's sampled meshes (span, pitch, axial nodes)
SAMPLED = [(41, 41, 97), (49, 49, 129), (65, 65, 161)]


def _solve(name, geometry, mesh, precision, points=1, multigrid=True, variant="default", cycles=20, kind="solve"):
    """mesh: "IMxJMxKM", or "sampled" for the three sampled meshes in turn"""
    return {"name": name, "kind": kind, "geometry": geometry, "mesh": mesh, "precision": precision, "points": points,
            "multigrid": multigrid, "variant": variant, "cycles": cycles}


def listed():
    return [
        # the smallest solve of the tests: latency and launches are all there is
        _solve("rotor 9x9x33 fp64", "rotor", "9x9x33", "fp64", multigrid=False),
        # the plain method: the annular duct, single grid
        _solve("duct 33x33x65 fp64", "duct", "33x33x65", "fp64", multigrid=False),
        # the benchmark's passage in the reference's precision
        _solve("rotor 49x49x129 fp64", "rotor", "49x49x129", "fp64"),
        # the same in the mixed form
        _solve("rotor 49x49x129 mixed", "rotor", "49x49x129", "mixed"),
        # a speed line on the mesh that converges: one batch, as speedline.run steps it
        _solve("speedline 32 x 25x25x65 mixed", "rotor", "25x25x65", "mixed", points=32, cycles=10),
        # operating points on meshes of uneven size in one batch, the largest work here
        _solve("batch 12 sampled mixed", "rotor", "sampled", "mixed", points=12, cycles=10),
        # odd, ragged mesh and the split-flux options, through the call surface
        _solve("rotor 35x27x52 fp64 sw calls", "rotor", "35x27x52", "fp64", multigrid=False, variant="sw_nnd",
               cycles=10, kind="calls"),
        # the central scheme, two grid levels
        _solve("rotor 25x33x65 fp64 jst", "rotor", "25x33x65", "fp64", variant="jst"),
        # the one-equation turbulence model
        _solve("rotor 49x49x129 mixed sa", "rotor", "49x49x129", "mixed", multigrid=False, variant="sa"),
        # a rotor and a stator joined by a mixing plane
        _solve("stage 33x33x97 mixed", "stage", "33x33x97", "mixed"),
        # warm start: training, and the network on new rows
        {"name": "train 32768 rows", "kind": "train", "rows": 32768, "steps": 20},
        {"name": "infer 262144 rows", "kind": "infer", "rows": 262144},
    ]


def _log_uniform(rng, lo, hi):
    return lo * (hi / lo) ** rng.random()


def draw(rng):
    kind = rng.choice(["solve"] * 5 + ["calls", "train", "infer"])
    if kind == "train":
        return {"kind": kind, "rows": int(_log_uniform(rng, 1024, 32768)), "steps": rng.randint(5, 20)}
    if kind == "infer":
        return {"kind": kind, "rows": int(_log_uniform(rng, 100, 262144))}
    geometry = rng.choice(["rotor", "rotor", "rotor", "duct", "stage"])
    variant = rng.choice(["default", "default", "default", "sw_nnd", "cons_laminar", "jst", "sa"])
    if geometry == "stage":
        variant = "default"
    multigrid = variant != "sa" and rng.random() < 0.5
    if multigrid:       # even cell counts, patches on even cells
        im, jm = (2 * int(_log_uniform(rng, 4, 24)) + 1 for _ in range(2))
        km = 8 * int(_log_uniform(rng, 4, 16)) + 1
    else:
        im, jm = (int(_log_uniform(rng, 9, 49)) for _ in range(2))
        km = int(_log_uniform(rng, 33, 129))
    precision = rng.choice(["fp64", "mixed"])
    points = 1
    if geometry == "rotor" and kind == "solve":
        room = 12 * 256000 / (im * jm * km)
        points = max(1, min(32, int(_log_uniform(rng, 1, max(1.0, room))))) if precision == "mixed" else rng.choice([1, 1, 3])
    c = _solve(None, geometry, "%dx%dx%d" % (im, jm, km), precision, points, multigrid, variant, rng.randint(5, 20 if precision == "fp64" else 10), kind)
    del c["name"]
    return c


# ---- inputs ----------------------------------------------------------------------------------------
_TEMPLATES = {}     # case directories written once per process: the text grids are slow to format
_ROOT = None


def _root():
    global _ROOT
    if _ROOT is None:
        _ROOT = tempfile.TemporaryDirectory(prefix="gbturbo_cases_")
    return _ROOT.name


def _meshes(case):
    if case["mesh"] == "sampled":
        return [SAMPLED[q % len(SAMPLED)] for q in range(case["points"])]
    return [tuple(int(v) for v in case["mesh"].split("x"))] * case["points"]


def _template(geometry, mesh, multigrid, variant):
    key = (geometry, mesh, multigrid, variant)
    if key not in _TEMPLATES:
        options = dict(VARIANTS[variant], Ma0="0.45")
        if multigrid:
            options.update(multigrid="Y", coarse_iter="2")
        im, jm, km = mesh
        d = os.path.join(_root(), "t%d" % len(_TEMPLATES))
        if geometry == "stage":
            # the stator's row behind the rotor's, half as long
            km2 = 8 * max(2, km // 16) + 1
            case = meshgen.stage_passage(IM=im, JM1=jm, KM1=km, JM2=jm, KM2=km2, options=options)
            meshgen.write_multiblock_case(case, d)
        elif geometry == "duct":
            meshgen.write_case(meshgen.annular_duct(IM=im, JM=jm, KM=km, options=options), d)
        else:
            meshgen.write_case(meshgen.rotor_passage(IM=im, JM=jm, KM=km, options=options), d)
        _TEMPLATES[key] = d
    return _TEMPLATES[key]


def _points(case, seed):
    """One case directory per operating point; the seed draws the back pressures."""
    rng = np.random.default_rng(seed)
    lo, hi = (0.90, 0.94) if case["geometry"] == "duct" else (1.05, 1.25)
    dirs, root = [], tempfile.mkdtemp(prefix="points_", dir=_root())
    for q, mesh in enumerate(_meshes(case)):
        t = _template(case["geometry"], mesh, case["multigrid"], case["variant"])
        dirs += speedline.make_points(t, [rng.uniform(lo, hi)], os.path.join(root, "op%d" % q), ratio_of="Ptin")
    return dirs


def prepare(case, seed):
    if case["kind"] == "infer":
        weights, features = _network(case, seed)
        w = gbturbo.WarmStart()
        w.set_params(weights)
        return {"case": case, "net": w, "features": features}
    if case["kind"] == "train":
        # the fields of four operating points a few cycles into their solves
        some = _solve("", "rotor", "25x25x65", "mixed", points=4)
        w = gbturbo.WarmStart(seed=seed % 1000003)
        with gbturbo.Solver(_points(some, seed), gbturbo.MIXED) as s:
            s.init_uniform()
            s.iterate(20, history=False)
            params = np.random.default_rng(seed).normal(size=(4, gbturbo.WS_PARAMS))
            w.add_solves(s, params)
        w.train(1, case["rows"])            # fixes the normalisation
        return {"case": case, "net": w}
    s = gbturbo.Solver(_points(case, seed), gbturbo.FP64 if case["precision"] == "fp64" else gbturbo.MIXED)
    s.init_uniform()
    rng = np.random.default_rng(seed)
    for q in range(s.n_slots):
        s.set_cv(_field(s, q, rng), q)
    s.start_from_fine_state()
    return {"case": case, "solver": s}


#: the network's layers: inputs, five hidden layers, outputs
WIDTHS = [gbturbo.WS_IN, 256, 256, 256, 256, 256, gbturbo.WS_OUT]


def _network(case, seed):
    """Weights and biases, layer after layer, and rows of inputs: sines and cosines, coordinates, case
    parameters, and zeros in the columns that are not used."""
    rng = np.random.default_rng(seed)
    p = [np.concatenate([rng.normal(0.0, (2.0 / k) ** 0.5, size=n * k), rng.normal(0.0, 0.05, size=n)])
         for k, n in zip(WIDTHS[:-1], WIDTHS[1:])]
    f = rng.uniform(-1.0, 1.0, size=(case["rows"], gbturbo.WS_IN)).astype(np.float32)
    f[:, 54:] = 0.0
    return np.concatenate(p).astype(np.float32), f


def _field(s, slot, rng):
    """A starting field as another solve or a network gives it: the uniform start with boundary layers on
    the four passage walls, swirl, and smooth variations that the seed draws. (From the uniform start itself
    the first cycles' vorticity is rounding noise, and which point of a wall line Baldwin-Lomax picks hangs
    on its last bit.)"""
    im, jm, km, levels = s.dims(slot, 1)
    coarse = s.get("cv", slot, levels)
    rho, _, _, mz, e = coarse[tuple(n // 2 for n in coarse.shape[:3])]
    x, y, z = np.meshgrid(*((np.arange(n - 1) + 0.5) / (n - 1) for n in (im, jm, km)), indexing="ij")

    def wave():
        a, f, p = rng.uniform(-1, 1, size=4), rng.uniform(0.4, 1.6, size=(4, 3)), rng.uniform(0, 2 * np.pi, size=4)
        return sum(a[m] * np.sin(np.pi * (f[m, 0] * x + f[m, 1] * y + f[m, 2] * z) + p[m]) for m in range(4))

    speed, kinetic = mz / rho, 0.5 * mz * mz / rho
    profile = (1 - 0.5 * (2 * x - 1) ** 8) * (1 - 0.5 * (2 * y - 1) ** 8)
    r = rho * (1 + 0.02 * wave())
    u = speed * (0.12 + 0.03 * wave()) * profile
    v = speed * (0.25 + 0.05 * wave()) * profile
    w = speed * (1 + 0.04 * wave()) * profile
    energy = (e - kinetic) * (1 + 0.02 * wave()) + 0.5 * r * (u * u + v * v + w * w)
    return np.stack([r, r * u, r * v, r * w, energy], axis=-1)


# ---- one pass ---------------------------------------------------------------------------------------
def run(state):
    case = state["case"]
    if case["kind"] == "infer":
        return {"outputs": state["net"].forward(state["features"])}
    if case["kind"] == "train":
        loss = state["net"].train(case["steps"], case["rows"])
        return {"loss": np.float32(loss), "params": state["net"].get_params()}
    s = state["solver"]
    if case["kind"] == "calls":
        rows = []
        for _ in range(case["cycles"]):
            s.solver_step()
            rows.append(s.integrals())
        report = np.stack(rows)
    else:
        report = s.iterate(case["cycles"])
    # the norms of the cross-stream momenta are left out: they are sums of relative changes of components
    # that pass through zero, so the cell nearest to zero sets them and the last bit of that cell
    report = report[..., [0, 1, 2, 3, 4] if case["kind"] == "calls" else [0, 1, 5, 6, 7, 8, 9, 10, 11]]
    slots = range(s.n_slots)
    if case["precision"] == "fp64":
        return {"report": report, "field": [s.get("cv", q) for q in slots]}
    # the mixed form holds the primitive variables, and forms what the report sums, in 32 bits
    return {"report": report.astype(np.float32), "field": [s.get("pv", q).astype(np.float32) for q in slots]}


def work(case):
    if case["kind"] in ("infer", "train"):
        weights = sum(a * b for a, b in zip(WIDTHS[:-1], WIDTHS[1:]))
        n = case["rows"]
        if case["kind"] == "infer":
            return {"bytes": n * 4 * (gbturbo.WS_IN + gbturbo.WS_OUT), "flops": 2.0 * weights * n}
        # per step: a minibatch of samples in; weights, both moments in and out
        return {"bytes": case["steps"] * (n * 4 * 12 + weights * 4 * 6), "flops": 6.0 * weights * n * case["steps"]}
    cells = 0
    for im, jm, km in _meshes(case):
        cells += (im - 1) * (jm - 1) * (km - 1)
        if case["geometry"] == "stage":
            cells += (im - 1) * (jm - 1) * 8 * max(2, km // 16)
    w = 8 if case["precision"] == "fp64" else 4
    # a cycle reads and writes Q (64 bits in both forms) and reads the geometry of every cell and face
    # once (three faces of 23 values, a cell of 13); at the end one field goes out
    per_cell = 2 * 5 * 8 + (3 * 23 + 13) * w
    # fluxes of three faces (twice a cycle with two grid levels), two sweeps
    ops = 3 * 750 * (2 if case["multigrid"] else 1) + 2 * 350
    return {"bytes": case["cycles"] * cells * per_cell + cells * 6 * w, "flops": float(case["cycles"] * cells * ops)}


def exact(case, seed):
    """The network's outputs in 64 bits. The solves have none here: a cycle of the solver in numpy would
    restate the whole of it."""
    if case["kind"] != "infer":
        return None
    p, f = _network(case, seed)
    p, h, at = p.astype(np.float64), f.astype(np.float64), 0
    for layer, (k, n) in enumerate(zip(WIDTHS[:-1], WIDTHS[1:])):
        weight = p[at:at + n * k].reshape(n, k)
        bias = p[at + n * k:at + n * k + n]
        at += n * k + n
        z = h @ weight.T + bias
        h = z / (1.0 + np.exp(-z)) if layer < len(WIDTHS) - 2 else z
    return {"outputs": h}
