"""The calls whose speed this framework is judged by: forward models, objective gradients, Jacobian
rows, unit responses, constraint gradients and the warm-start network, each through the Python API.

`listed()` names the cases, `draw(rng)` makes further ones over the same ranges, `prepare` builds what
a program holds before the call (the context with its model and data, the parameters), `run` makes the
call, `work` counts what the call cannot do without, and `exact` restates the call in plain 64-bit
torch.  Geometry follows from the case alone; parameters, properties, station positions and
observations follow from the seed.
"""
import functools
import math

import numpy as np
import torch

from lithoinv3d_b200 import synth
from lithoinv3d_b200.api import (COLLAPSED_DROP, FIXED, GATHER_CHAIN, GRAVITY, MAGNETIC, PREC_FP64, PREC_MIXED,
                                 UNIT_GRAVITY, UNIT_INDUCED, XY_FORWARD_DIFFERENCE, XYZ_FREE, Z_ONLY)
from lithoinv3d_b200.warmstart import Network

INDUCING = (60.0, 10.0, 55000.0)  # inclination and declination (degrees), field (nT)
FD_STEP = 0.5  # metres, of the finite-difference XY derivative
GAL = 6.67430e-11 * 1e3 * 1e5  # mGal per g/cc

# Flops per (station, facet) pair, special functions as one each: the facet terms of gz and TMI, and their
# derivatives by the facet's nine vertex coordinates contracted with the two adjoints.
FORWARD_FLOPS, GRADIENT_FLOPS = 148, 344


def listed():
    return [
        # A single body under a small survey, FP64 (the default precision): the smallest call, bound by latency.
        dict(name="body_forward", kind="forward", model="icosphere", level=2, side=23, precision="fp64"),
        # The single-body inversion: objective and gradient, once per L-BFGS iteration, FP64.
        dict(name="body_gradient", kind="gradient", model="icosphere", level=3, side=40, precision="fp64"),
        # Dense sensitivity rows of the same body, as Gauss-Newton steps and resolution studies take them.
        dict(name="body_jacobian", kind="jacobian", model="icosphere", level=3, side=40, which="gravity"),
        # The contact-model inversion: control points every 4th vertex, joint gz + TMI, mixed precision, the
        # evaluation replayed as a graph: what one iteration of a production run costs.
        dict(name="contact_gradient_mixed", kind="gradient", model="contact", nx=24, ny=24, nz=12, groups=4, blobs=6,
             geometry=3, cp=4, side=64, precision="mixed", graph=True),
        # The same kind of model at full resolution in FP64, on odd sizes.
        dict(name="contact_gradient_fp64", kind="gradient", model="contact", nx=21, ny=19, nz=11, groups=3, blobs=5,
             geometry=4, cp=0, side=57, precision="fp64"),
        # Forward modelling of a survey whose gravity and magnetic stations differ (a ground grid and a denser
        # airborne one), mixed precision.
        dict(name="survey_forward_mixed", kind="forward", model="contact", nx=27, ny=20, nz=9, groups=5, blobs=8,
             geometry=5, cp=0, side=37, mag_side=101, precision="mixed"),
        # The columns of the property inversion: every group's unit gravity and unit susceptibility response.
        dict(name="property_columns", kind="unit", model="contact", nx=24, ny=24, nz=12, groups=4, blobs=6,
             geometry=3, cp=0, side=64, precision="fp64"),
        # The large single inversion: x/y/z-free vertices under topography, exact chain gradient, collapsed
        # facets dropped; the largest call.
        dict(name="large_gradient_mixed", kind="gradient", model="large", nx=60, ny=60, nz=30, groups=6, blobs=20,
             geometry=5, cp=4, side=200, precision="mixed", graph=True),
        # Many independent bodies in one evaluation, uneven facet and station counts.
        dict(name="batch_gradient_mixed", kind="gradient", model="batch", bodies=32, geometry=21, precision="mixed",
             graph=True),
        # The large configuration's half-metre finite-difference XY derivatives, on a model without control points.
        dict(name="fdxy_gradient", kind="gradient", model="large", nx=14, ny=13, nz=8, groups=3, blobs=6, geometry=7,
             cp=0, side=45, precision="fp64", xy="fd"),
        # Borehole constraints: the finite-difference gradient of the classification penalty.
        dict(name="constraint_gradient", kind="constraints", model="contact", nx=24, ny=24, nz=12, groups=4, blobs=6,
             geometry=3, cp=4, intervals=64),
        # The warm-start network: some batches of training, then its weights read back as a checkpoint.
        dict(name="network_training", kind="network", inputs=8192, outputs=1313, width=512, depth=4, batch=256,
             batches=32),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def contact(lo, hi, **more):
        return dict(model="contact", nx=rng.randint(lo, hi), ny=rng.randint(lo, hi), nz=rng.randint(5, 13),
                    groups=rng.randint(2, 6), blobs=rng.randint(4, 9), geometry=rng.randint(1, 99), **more)

    kind = rng.choice(["body", "body", "jacobian", "contact", "contact", "full", "survey", "unit", "large", "batch",
                       "fdxy", "constraints", "network"])
    if kind == "body":
        return dict(kind=rng.choice(["forward", "gradient"]), model="sphere", lat=log_int(6, 48), lon=log_int(8, 64),
                    side=log_int(12, 64), precision=rng.choice(["fp64", "fp64", "mixed"]))
    if kind == "jacobian":
        return dict(kind="jacobian", model="sphere", lat=log_int(6, 24), lon=log_int(8, 32), side=log_int(12, 40),
                    which=rng.choice(["gravity", "magnetic"]))
    if kind == "contact":
        return dict(kind="gradient", cp=rng.choice([0, 4]), side=log_int(30, 72), graph=True,
                    precision=rng.choice(["mixed", "mixed", "fp64"]), **contact(12, 28))
    if kind == "full":
        return dict(kind="gradient", cp=0, side=log_int(24, 64), precision="fp64", **contact(12, 26))
    if kind == "survey":
        return dict(kind="forward", cp=0, side=log_int(20, 60), mag_side=log_int(40, 128),
                    precision=rng.choice(["fp64", "mixed"]), **contact(12, 30))
    if kind == "unit":
        return dict(kind="unit", cp=0, side=log_int(24, 72), precision=rng.choice(["fp64", "mixed"]), **contact(12, 26))
    if kind == "large":
        n = rng.randint(24, 48)
        return dict(kind="gradient", model="large", nx=n, ny=rng.randint(20, n), nz=rng.randint(10, 24),
                    groups=rng.randint(3, 7), blobs=rng.randint(8, 20), geometry=rng.randint(1, 99),
                    cp=rng.choice([0, 4]), side=log_int(60, 160), precision="mixed", graph=True)
    if kind == "batch":
        return dict(kind="gradient", model="batch", bodies=rng.randint(6, 30), geometry=rng.randint(1, 99),
                    precision="mixed", graph=True)
    if kind == "fdxy":
        return dict(kind="gradient", model="large", nx=rng.randint(8, 15), ny=rng.randint(8, 15),
                    nz=rng.randint(4, 9), groups=rng.randint(2, 4), blobs=rng.randint(3, 7),
                    geometry=rng.randint(1, 99), cp=0, side=log_int(24, 50), precision=rng.choice(["fp64", "mixed"]),
                    xy="fd")
    if kind == "constraints":
        return dict(kind="constraints", cp=4, intervals=log_int(16, 128), **contact(14, 24))
    return dict(kind="network", inputs=2 * log_int(400, 4096), outputs=log_int(200, 1500),
                width=128 * rng.randint(1, 5), depth=rng.randint(2, 5), batch=128 * rng.randint(1, 3),
                batches=rng.randint(4, 32))


# ---------------------------------------------------------------- geometry --
# Plain arrays, the same for every seed: kept between preparations (they are never written to).


@functools.lru_cache(maxsize=8)
def _meshes(model, size, geometry):
    """[(vertices, triangles, freedoms)] per group, and for batched bodies their station grids."""
    if model == "icosphere":
        U, F = synth.icosphere(size[0])
        return [(U * 200.0 + [0.0, 0.0, -500.0], F, np.full(len(U), Z_ONLY, np.uint8))], None
    if model == "sphere":
        U, F = synth.latlong_sphere(*size)
        return [(U * 200.0 + [0.0, 0.0, -500.0], F, np.full(len(U), Z_ONLY, np.uint8))], None
    if model == "batch":
        p = synth.batch_bodies_model(n_bodies=size[0], seed=geometry)
        edges = np.cumsum([0] + list(p.station_groups))
        return ([(V, F, np.full(len(V), fr, np.uint8)) for V, F, fr in p.meshes],
                [p.grav_xyz[a:b] for a, b in zip(edges[:-1], edges[1:])])
    nx, ny, nz, groups, blobs = size
    large = model == "large"
    p = synth.voxel_contact_model(shape=(nx, ny, nz), n_groups=groups, n_blobs=blobs, seed=geometry, n_side=4,
                                  freedom_interior=XYZ_FREE if large else Z_ONLY,
                                  blob_width=(0.05, 0.15) if large and nx > 40 else (0.1, 0.3))
    return [m for m in p.meshes if len(m[1])], None


def _geometry(case):
    m = case["model"]
    size = {"icosphere": ("level",), "sphere": ("lat", "lon"), "batch": ("bodies",)}.get(
        m, ("nx", "ny", "nz", "groups", "blobs"))
    return _meshes(m, tuple(case[k] for k in size), case.get("geometry", 0))


def _footprint(case):
    return (2000.0, 2000.0) if case["model"] in ("icosphere", "sphere") else (100.0 * case["nx"], 100.0 * case["ny"])


def _grid_shape(case, side):
    w, h = _footprint(case)
    return side, max(2, int(round(side * h / w)))


def _stations(case, side, rng):
    """A survey over the footprint: a grid with a tenth of its spacing of navigation scatter, 1 m above the
    flat surface, or above topography on the large model."""
    n, m = _grid_shape(case, side)
    w, _ = _footprint(case)
    st = synth.station_grid(n, w / n, 1.0, ny=m)
    st[:, :2] += rng.uniform(-0.1, 0.1, (len(st), 2)) * (w / n)
    if case["model"] == "large":
        st[:, 2] += synth.topography(st[:, :2], rng)
    return st


def _anomaly(st, rng, amplitude):
    """Observations: a smooth anomaly and one per cent of noise; and their standard deviations."""
    span = float(np.max(np.ptp(st[:, :2], axis=0))) or 1.0
    v = np.zeros(len(st))
    for _ in range(6):
        c = st[rng.integers(len(st)), :2]
        v += rng.normal() * np.exp(-((st[:, :2] - c) ** 2).sum(1) / (2 * (rng.uniform(0.1, 0.3) * span) ** 2))
    v *= amplitude / (np.std(v) + 1e-12)
    sd = 0.01 * np.std(v)
    return v + rng.normal(0.0, sd, len(v)), np.full(len(v), sd)


def _inputs(case, seed):
    """Everything of a case that depends on the seed, as numpy arrays."""
    rng = np.random.default_rng([seed, 77])
    meshes, grids = _geometry(case)
    d = dict(rho=rng.uniform(0.1, 0.5, len(meshes)) * rng.choice([-1.0, 1.0], len(meshes)),
             chi=rng.uniform(0.005, 0.05, len(meshes)))
    if grids is not None:
        st = np.concatenate(grids)
        st = st + np.concatenate([rng.uniform(-1.0, 1.0, (len(st), 2)), np.zeros((len(st), 1))], axis=1)
        d["grav"] = d["mag"] = st
    elif case["kind"] == "constraints":
        d["grav"] = d["mag"] = np.array([[0.0, 0.0, 1.0]])
    else:
        d["grav"] = _stations(case, case["side"], rng)
        d["mag"] = _stations(case, case["mag_side"], rng) if "mag_side" in case else d["grav"]
    if case["kind"] == "gradient":
        d["gobs"], d["gsd"] = _anomaly(d["grav"], rng, 3.0)
        d["mobs"], d["msd"] = _anomaly(d["mag"], rng, 100.0)
    d["step"] = rng  # drawn from further, in order, once the number of parameters is known
    return d


def _model(case, d):
    meshes, grids = _geometry(case)
    z = np.zeros((1, 3))
    return synth.Problem(case["model"], list(d["rho"]), list(d["chi"]), meshes, z, z, cp_stride=case.get("cp", 0),
                         station_groups=None if grids is None else [len(g) for g in grids]).build_model()


def _perturbed(case, x0, rng):
    """Parameters of an iterate: a few metres off the start model."""
    return x0 + rng.normal(0.0, 2.0 if case["model"] == "large" else 5.0, len(x0))


def _network_inputs(case, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = case["batch"] * case["batches"]
    X = torch.randn((n, case["inputs"]), generator=g, device="cuda")
    Y = torch.randn((n, case["outputs"]), generator=g, device="cuda")
    return X, Y


# ------------------------------------------------------------ the calls --


def prepare(case, seed):
    if case["kind"] == "network":
        net = Network(case["inputs"], case["outputs"], width=case["width"], depth=case["depth"], batch=case["batch"],
                      seed=seed)
        X, Y = _network_inputs(case, seed)
        i, w, o = case["inputs"], case["width"], case["outputs"]
        weights = np.empty(i * w + w + (case["depth"] - 1) * (w * w + w) + w * o + o, np.float32)
        return dict(case=case, net=net, X=X, Y=Y, weights=weights, order=seed)
    d = _inputs(case, seed)
    model = _model(case, d)
    x = _perturbed(case, model.assemble_parameters(), d["step"])
    ctx = synth.Context(0)
    ctx.set_model(model)
    if case["model"] == "batch":
        ctx.set_station_groups([len(g) for g in _geometry(case)[1]])
    ctx.set_field(*INDUCING)
    ctx.set_gravity_data(d["grav"], d.get("gobs"), d.get("gsd"))
    ctx.set_magnetic_data(d["mag"], d.get("mobs"), d.get("msd"))
    ctx.set_precision(PREC_MIXED if case.get("precision") == "mixed" else PREC_FP64)
    ctx.set_scatter_stateless(True)  # each evaluation a function of its parameters alone
    if case["model"] == "large":
        ctx.set_collapsed_facets(COLLAPSED_DROP)
        if case.get("cp"):
            ctx.set_gradient_gather(GATHER_CHAIN)
    if case.get("xy") == "fd":
        ctx.set_xy_derivative(XY_FORWARD_DIFFERENCE, FD_STEP)
    if case.get("graph"):
        ctx.set_graph_mode(True)
    if case["kind"] == "constraints":
        model.apply_parameters(x)
        ctx.set_constraints(*_intervals(case, model, d["step"]))
    return dict(case=case, ctx=ctx, x=x, groups=len(d["rho"]))


def _intervals(case, model, rng):
    """Borehole intervals: half of the midpoints 0.3 m off control-point vertices, so that a one-metre step of
    that vertex changes their class, the others anywhere in the model."""
    t = model.tables()
    cps = np.unique(t["ref_vertex"][t["ref_axis"] == 2])
    near = min(case["intervals"] // 2, len(cps))
    mid = model.positions()[rng.choice(cps, near, replace=False)] + np.where(rng.random((near, 1)) < 0.5, 0.3, -0.3) * [0, 0, 1]
    w, h = _footprint(case)
    far = rng.uniform([-0.48 * w, -0.48 * h, -95.0 * case["nz"]], [0.48 * w, 0.48 * h, -20.0],
                      (case["intervals"] - near, 3))
    mid = np.concatenate([mid, far])
    half = rng.uniform(0.5, 40.0, len(mid))
    return mid[:, :2].copy(), -mid[:, 2] - half, -mid[:, 2] + half, rng.integers(0, case["groups"], len(mid))


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "forward":
        gz, tmi = s["ctx"].forward(s["x"])
        return {"gz": gz, "tmi": tmi}
    if kind == "gradient":
        f, g = s["ctx"].objective_and_gradient(s["x"])
        return {"f": np.array(f), "gradient": g}
    if kind == "jacobian":
        return s["ctx"].jacobian(s["x"], GRAVITY if case["which"] == "gravity" else MAGNETIC)
    if kind == "unit":
        return [s["ctx"].unit_response(s["x"], k, g) for k in (UNIT_GRAVITY, UNIT_INDUCED) for g in range(s["groups"])]
    if kind == "constraints":
        return s["ctx"].constraint_gradient(s["x"])
    net = s["net"]
    losses = net.train(s["X"], s["Y"], epochs=1, lr=1e-3, rng=np.random.default_rng(s["order"]))
    net.lib.lf_mlp_get_params(net.h, s["weights"].ctypes.data)
    return {"loss": np.array(losses), "weights": s["weights"]}


def work(case):
    if case["kind"] == "network":
        i, w, o, n = case["inputs"], case["width"], case["outputs"], case["batch"] * case["batches"]
        weights = i * w + (case["depth"] - 1) * w * w + w * o
        return {"bytes": 4 * n * (i + o) + 4 * weights + 24 * weights * case["batches"],
                "flops": 6 * n * weights - 2 * n * i * w}
    meshes, grids = _geometry(case)
    facets = sum(len(F) for _, F, _ in meshes)
    vertices = sum(len(V) for V, _, _ in meshes)
    free, moved = _moved(case)
    kind = case["kind"]
    if kind == "constraints":  # two classifications of every interval per parameter: a sign test per facet
        n = int(free)
        return {"bytes": 24 * vertices + 12 * facets + 8 * n, "flops": 2 * n * case["intervals"] * facets * 4}
    if grids is not None:
        counts = [len(g) for g in grids]
        pairs = sum(c * len(F) for c, (_, F, _) in zip(counts, meshes))
        stations = 2 * sum(counts)
        grad = pairs
    else:
        def count(side):
            n, m = _grid_shape(case, side)
            return n * m

        g = count(case["side"])
        m = count(case["mag_side"]) if "mag_side" in case else g
        stations = g + m
        pairs, grad = 0.5 * (g + m) * facets, 0.5 * (g + m) * moved
    geometry = 24 * vertices + 12 * facets + 24 * stations
    if kind == "forward":
        return {"bytes": geometry + 8 * stations, "flops": FORWARD_FLOPS * pairs}
    if kind == "unit":
        return {"bytes": len(meshes) * (geometry + 8 * stations), "flops": FORWARD_FLOPS * pairs}
    if kind == "jacobian":
        return {"bytes": geometry + 4 * stations * free, "flops": 0.5 * GRADIENT_FLOPS * grad}
    flops = FORWARD_FLOPS * pairs + GRADIENT_FLOPS * grad
    if case.get("xy") == "fd":
        flops += 6 * FORWARD_FLOPS * grad
    return {"bytes": geometry + 16 * stations + 16 * free, "flops": flops}


@functools.lru_cache(maxsize=64)
def _moved_of(key):
    """(number of parameters, facets with a vertex whose derivative is asked for)."""
    case = dict(key)
    meshes, _ = _geometry(case)
    model = _model(case, dict(rho=np.ones(len(meshes)), chi=np.ones(len(meshes))))
    t = model.tables()
    on = np.zeros(len(t["pos"]), bool)
    on[t["ref_vertex"]] = True
    if case["model"] == "large" and case.get("cp"):
        on |= np.diff(t["interp_off"]) > 0
    return model.n_dofs, int(on[t["tri"]].any(axis=1).sum())


def _moved(case):
    return _moved_of(tuple(sorted(case.items())))


# --------------------------------------------------------- plain 64 bits --
# gz and TMI of a triangle at a station (Nagy's facet sum; the TMI facet term with the solid angle and the three
# edge integrals), written component by component; everything below is torch float64.


def _facet_terms(a, b, c, o, mdir, fdir):
    """Unscaled facet terms of gz and TMI, [facets, stations].  a, b, c: vertex components, each [facets, 1] (or
    [facets, stations]); o: station components [1, stations]; mdir [facets][3], fdir [3]."""
    def sub(u, v):
        return [x - y for x, y in zip(u, v)]

    def dot(u, v):
        return u[0] * v[0] + u[1] * v[1] + u[2] * v[2]

    def cross(u, v):
        return [u[1] * v[2] - u[2] * v[1], u[2] * v[0] - u[0] * v[2], u[0] * v[1] - u[1] * v[0]]

    n = cross(sub(b, a), sub(c, a))
    size = torch.sqrt(dot(n, n))
    un = [x / size for x in n]
    r = [sub(p, o) for p in (a, b, c)]
    d = [torch.sqrt(dot(p, p)) for p in r]
    num = dot(r[0], cross(r[1], r[2]))
    den = d[0] * d[1] * d[2] + dot(r[0], r[1]) * d[2] + dot(r[0], r[2]) * d[1] + dot(r[1], r[2]) * d[0]
    omega = 2.0 * torch.atan2(num, den)
    gz = -dot(r[0], un) * omega
    tmi = dot(mdir, un) * dot(fdir, un) * omega
    corners = (a, b, c)
    for i in range(3):
        j = (i + 1) % 3
        e = sub(corners[j], corners[i])
        L = torch.sqrt(dot(e, e))
        perp = cross(un, [x / L for x in e])
        lam = torch.log1p(2.0 * L / (d[i] + d[j] - L))
        gz = gz - dot(r[i], perp) * lam
        tmi = tmi + dot(mdir, perp) * dot(fdir, perp) * lam
    return un[2] * gz, tmi


def _direction():
    i, k = math.radians(INDUCING[0]), math.radians(INDUCING[1])
    return [math.cos(i) * math.cos(k), math.cos(i) * math.sin(k), -math.sin(i)]


def _parameters(meshes):
    """The parameter of every (vertex, axis) it writes: arrays vertex, axis, parameter, and the start values.
    Free coordinates at the same micrometre-rounded position and axis are one parameter, numbered by first
    appearance over groups, vertices and axes."""
    axes = {FIXED: (), Z_ONLY: (2,), XYZ_FREE: (0, 1, 2)}
    vertex, axis, keys, start, base = [], [], [], [], 0
    for V, _, fr in meshes:
        v = np.repeat(np.arange(len(V)), [len(axes[f]) for f in fr])
        ax = np.concatenate([np.array(axes[f], int) for f in fr]) if len(v) else np.zeros(0, int)
        q = (np.sign(V) * np.floor(np.abs(V * 1e6) + 0.5)).astype(np.int64).view(np.uint64)
        keys.append(q[v, 0] ^ (q[v, 1] << np.uint64(21)) ^ (q[v, 2] << np.uint64(42))
                    ^ (ax.astype(np.uint64) << np.uint64(60)))
        vertex.append(v + base)
        axis.append(ax)
        start.append(V[v, ax])
        base += len(V)
    keys, start = np.concatenate(keys), np.concatenate(start)
    _, first, inv = np.unique(keys, return_index=True, return_inverse=True)
    order = np.argsort(first)
    rank = np.empty(len(order), int)
    rank[order] = np.arange(len(order))
    return np.concatenate(vertex), np.concatenate(axis), rank[inv.reshape(-1)], start[first[order]]


def _plain(case, d):
    """Vertices at the iterate, triangles and per-facet scales as device tensors."""
    meshes, _ = _geometry(case)
    vertex, axis, par, start = _parameters(meshes)
    x = _perturbed(case, start, d["step"])
    pos = np.concatenate([V for V, _, _ in meshes])
    pos[vertex, axis] = x[par]
    off = np.cumsum([0] + [len(V) for V, _, _ in meshes])
    tri = np.concatenate([F + o for (_, F, _), o in zip(meshes, off)])
    group = np.repeat(np.arange(len(meshes)), [len(F) for _, F, _ in meshes])
    dev = "cuda" if torch.cuda.is_available() else "cpu"

    def t(v, dtype=torch.float64):
        return torch.as_tensor(np.ascontiguousarray(v), dtype=dtype, device=dev)

    return dict(pos=t(pos), tri=t(tri, torch.int64), group=t(group, torch.int64), n=len(start),
                vertex=t(vertex, torch.int64), axis=t(axis, torch.int64), par=t(par, torch.int64),
                gscale=t(GAL * d["rho"]), mscale=t(-d["chi"] * INDUCING[2] / (4.0 * math.pi)),
                fdir=[t(v) for v in _direction()], t=t)


def _columns(v):
    return [v[:, k:k + 1] for k in range(3)]


def _sums(P, tri, group, st, ones=None):
    """Forward sums of gz and TMI of the given facets at stations st [n, 3]; ones: unit scales."""
    gz, tmi = torch.zeros(len(st), dtype=torch.float64, device=st.device), torch.zeros_like(st[:, 0])
    step = max(1, (1 << 21) // max(1, len(tri)))
    a, b, c = (_columns(P["pos"][tri[:, k]]) for k in range(3))
    gs = P["gscale"][group] if ones is None else torch.full_like(a[0][:, 0], ones[0])
    ms = P["mscale"][group] if ones is None else torch.full_like(a[0][:, 0], ones[1])
    for s in range(0, len(st), step):
        o = [v.T for v in _columns(st[s:s + step])]
        g, m = _facet_terms(a, b, c, o, P["fdir"], P["fdir"])
        gz[s:s + step], tmi[s:s + step] = gs @ g, ms @ m
    return gz, tmi


def _vertex_gradient(P, tri, group, st, cg, cm, fd):
    """d(sum_s cg gz + cm tmi) / d(vertex), [vertices, 3]; fd: x and y by forward differences of each facet."""
    out = torch.zeros_like(P["pos"])
    step = max(1, (1 << 20) // max(1, len(tri)))
    gs, ms = P["gscale"][group][:, None], P["mscale"][group][:, None]
    for s in range(0, len(st), step):
        o = [v.T for v in _columns(st[s:s + step])]
        wg, wm = gs * cg[None, s:s + step], ms * cm[None, s:s + step]
        corners = [P["pos"][tri[:, k]].clone().requires_grad_(True) for k in range(3)]
        g, m = _facet_terms(*(_columns(v) for v in corners), o, P["fdir"], P["fdir"])
        grads = list(torch.autograd.grad((wg * g + wm * m).sum(), corners))
        if fd:
            with torch.no_grad():
                for k in range(3):
                    for ax in range(2):
                        moved = [v.detach().clone() for v in corners]
                        moved[k][:, ax] += FD_STEP
                        g1, m1 = _facet_terms(*(_columns(v) for v in moved), o, P["fdir"], P["fdir"])
                        grads[k][:, ax] = (wg * (g1 - g) + wm * (m1 - m)).sum(1) / FD_STEP
        for k in range(3):
            out.index_add_(0, tri[:, k], grads[k])
    return out


def exact(case, seed):
    # None for the classification penalty (decisions, not arithmetic), for control-point models (the choice of the
    # control points is the framework's own), and where the sums would take too long.
    if case["kind"] == "constraints" or case.get("cp"):
        return None
    if case["kind"] == "network":
        return _exact_network(case)
    if work(case)["flops"] > 7e11:
        return None
    d = _inputs(case, seed)
    P = _plain(case, d)
    t = P["t"]
    meshes, grids = _geometry(case)
    if grids is None:
        parts = [(P["tri"], P["group"], slice(None))]
    else:  # each body sees its own stations
        fo = np.cumsum([0] + [len(F) for _, F, _ in meshes])
        so = np.cumsum([0] + [len(g) for g in grids])
        parts = [(P["tri"][fo[k]:fo[k + 1]], P["group"][fo[k]:fo[k + 1]], slice(so[k], so[k + 1]))
                 for k in range(len(meshes))]
    grav, mag = t(d["grav"]), t(d["mag"])
    if case["kind"] == "jacobian":
        return _exact_jacobian(case, P, grav if case["which"] == "gravity" else mag)
    if case["kind"] == "unit":
        unit = (GAL, -INDUCING[2] / (4.0 * math.pi))
        cols = [_sums(P, P["tri"][P["group"] == g], P["group"][P["group"] == g], grav, unit)
                for g in range(len(meshes))]
        return [c[0].cpu().numpy() for c in cols] + [c[1].cpu().numpy() for c in cols]
    gz, tmi = torch.zeros_like(grav[:, 0]), torch.zeros_like(mag[:, 0])
    for tri, group, sl in parts:
        g, m = _sums(P, tri, group, grav[sl])
        gz[sl] = g
        tmi[sl] = m if d["mag"] is d["grav"] else _sums(P, tri, group, mag[sl])[1]
    if case["kind"] == "forward":
        return {"gz": gz.cpu().numpy(), "tmi": tmi.cpu().numpy()}
    gobs, mobs, gw, mw = t(d["gobs"]), t(d["mobs"]), 1.0 / t(d["gsd"]), 1.0 / t(d["msd"])
    rg, rm = gw * (gobs - gz), mw * (mobs - tmi)
    f = 0.5 * (rg * rg).sum() + 0.5 * (rm * rm).sum()
    vg = torch.zeros_like(P["pos"])
    for tri, group, sl in parts:
        vg += _vertex_gradient(P, tri, group, grav[sl], -gw[sl] * rg[sl], -mw[sl] * rm[sl], case.get("xy") == "fd")
    grad = torch.zeros(P["n"], dtype=torch.float64, device=vg.device)
    grad.index_add_(0, P["par"], vg[P["vertex"], P["axis"]])
    return {"f": np.array(float(f)), "gradient": grad.cpu().numpy()}


def _exact_jacobian(case, P, st):
    J = torch.zeros((P["n"], len(st)), dtype=torch.float64, device=st.device)
    tri, group = P["tri"], P["group"]
    step = max(1, (1 << 20) // len(tri))
    column = torch.full((len(P["pos"]), 3), -1, dtype=torch.int64, device=st.device)
    column[P["vertex"], P["axis"]] = P["par"]
    for s in range(0, len(st), step):
        o = [v.T for v in _columns(st[s:s + step])]
        n = o[0].shape[1]
        corners = [[v.expand(-1, n).clone().requires_grad_(True) for v in _columns(P["pos"][tri[:, k]])]
                   for k in range(3)]
        g, m = _facet_terms(*corners, o, P["fdir"], P["fdir"])
        y = P["gscale"][group] @ g if case["which"] == "gravity" else P["mscale"][group] @ m
        grads = torch.autograd.grad(y.sum(), [v for k in corners for v in k])
        for k in range(3):
            for ax in range(3):
                col = column[tri[:, k], ax]
                J[:, s:s + n].index_add_(0, col[col >= 0], grads[3 * k + ax][col >= 0])
    return J.T.contiguous().cpu().numpy()


def _exact_network(case):
    # The network starts from the framework's own random weights, and Adam's first steps have the size of the
    # learning rate whatever the gradient's: no plain value to be held to.
    return None
