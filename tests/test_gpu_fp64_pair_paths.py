"""The FP64 forward's two routes per pair (polynomials away from the facet, the
reference's branches near it) at the lines between them, against the oracle.

Tolerance, per station: 256 eps x the sum of the magnitudes of the facet
terms.  Every term has a relative error of a few eps on either side; the
oracle's edge integral log((s2 + d2) / (s1 + d1)) loses up to a factor 17 in
s1 + d1 (stations at least 20 degrees off an edge's direction)."""
import numpy as np
import pytest

from lithoinv3d_b200 import GATHER_CHAIN, GRAVITY, MAGNETIC, synth
from lithoinv3d_b200.api import COLLAPSED_DROP
from oracle_bindings import OracleModel

pytestmark = pytest.mark.gpu

V = np.array([[0.0, 0.0, -100.0], [120.0, 0.0, -100.0], [0.0, 90.0, -100.0], [30.0, 20.0, -180.0]])
F = np.array([[0, 1, 2], [0, 3, 1], [1, 3, 2], [2, 3, 0]], np.int32)
EPS = np.finfo(float).eps


def at_edge_ratio(v):
    """Stations that see the edge 0-1 with L / (d1 + d2) = v, out of every facet's plane."""
    L = 120.0
    off = np.sqrt((L / (2 * v)) ** 2 - (L / 2) ** 2)
    th = np.radians([35.0, 62.0, 118.0])
    return np.stack([np.full(3, 60.0), -off * np.cos(th), -100.0 + off * np.sin(th)], axis=1)


def off_plane(rel):
    """Stations rel x their distance to vertex 0 above the plane of facet 0, 45 degrees off its edges."""
    d = np.array([-250.0, -1000.0, -4000.0])
    return np.stack([d, d, -100.0 + rel * np.abs(d) * np.sqrt(2.0)], axis=1)


CASES = {
    "quarter": np.concatenate([at_edge_ratio(0.25 * (1 + s)) for s in (-1e-3, -1e-9, 1e-9, 1e-3)]),
    "half": np.concatenate([at_edge_ratio(0.5 * (1 + s)) for s in (-1e-3, -1e-9, 1e-9, 1e-3)]),
    "close": np.concatenate([at_edge_ratio(v) for v in (0.7, 0.95, 0.999)]),
    "plane": np.concatenate([off_plane(s * 2.0 ** -k) for k in (19.5, 20.5, 30) for s in (1, -1)] + [off_plane(0.0)]),
    "vertex and edge line": np.array([V[0], V[1], [240.0, 0.0, -100.0], [-60.0, 0.0, -100.0], [60.0, 0.0, -100.0],
                                      [0.0, 4000.0, -100.0]]),
    "far": np.array([[1e6, -2e6, 5e5], [3e4, 0.0, 1.0], [-700.0, 900.0, 1.0]]),
}


def term_sums(sta, rho, chi, field):
    """Sum over facets of the magnitudes of the gz and TMI terms (scaled)."""
    g = 6.67430e-11 * 1e3 * 1e5 * abs(rho)
    m = abs(chi) * field[2] / (4 * np.pi)
    out = np.zeros((len(sta), 2))
    for f in F:
        p = V[f][None] - sta[:, None]
        d = np.linalg.norm(p, axis=2)
        lam = np.array([np.log1p(2 * L / np.maximum(d[:, i] + d[:, (i + 1) % 3] - L, 1e-12 * L))
                        for i, L in enumerate(np.linalg.norm(V[np.roll(f, -1)] - V[f], axis=1))])
        out[:, 0] += g * (d.max(1) * (lam.sum(0) + 2 * np.pi))
        out[:, 1] += m * (lam.sum(0) + 2 * np.pi)
    return out


@pytest.mark.parametrize("name", list(CASES))
def test_forward_routes(name):
    sta = CASES[name]
    p = synth.Problem("tetrahedron", [0.3], [0.02], [(V, F, synth.Z_ONLY)], sta, sta)
    model = p.build_model()
    ctx = p.make_context(model)
    x = model.assemble_parameters()
    gz, tmi = ctx.forward(x)
    om = OracleModel(model.tables(), p.densities, p.susceptibilities, p.inducing)
    om.scatter(x)
    tol = 256 * EPS * term_sums(sta, 0.3, 0.02, p.inducing)
    assert np.all(np.abs(gz - om.forward_gz(sta)) <= tol[:, 0])
    assert np.all(np.abs(tmi - om.forward_tmi(sta)) <= tol[:, 1])


@pytest.mark.parametrize("which", [GRAVITY, MAGNETIC])
@pytest.mark.parametrize("name", ["quarter", "half", "close"])
def test_derivative_routes(name, which):
    """Jacobian rows on both sides of the lines between the routes, against the
    oracle's central-difference truth (1e-6 of the row's largest entry, the
    tolerance of the other Jacobian tests)."""
    sta = CASES[name]
    p = synth.Problem("tetrahedron", [0.3], [0.02], [(V, F, synth.XYZ_FREE)], sta, sta)
    model = p.build_model()
    ctx = p.make_context(model)
    x = model.assemble_parameters()
    J = ctx.jacobian(x, which)
    om = OracleModel(model.tables(), p.densities, p.susceptibilities, p.inducing)
    om.scatter(x)
    Jt = om.jacobian(sta, 2 + which)
    assert np.all(np.abs(J - Jt).max(1) <= 1e-6 * np.abs(Jt).max(1))


def test_one_data_type_gradient():
    """The gradient kernels for gravity or magnetic data alone against the sum
    they split: the joint gradient is linear in the adjoints, and each station
    set's part is computed by the kernel of its own (64 eps of the joint
    gradient's largest entry per entry, several times the rounding of sums over
    9 stations and 4 facets)."""
    rng = np.random.default_rng(3)
    sta = np.concatenate([CASES["quarter"], CASES["far"][1:]]) + rng.uniform(-1.0, 1.0, (14, 3))
    p = synth.Problem("tetrahedron", [0.3], [0.02], [(V, F, synth.XYZ_FREE)], sta, sta)
    model = p.build_model()
    ctx = p.make_context(model)
    x = model.assemble_parameters()
    joint = ctx.objective_and_gradient(x)[1]
    none = np.zeros((0, 3))
    ctx.set_magnetic_data(none)
    grav = ctx.objective_and_gradient(x)[1]
    ctx.set_gravity_data(none)
    ctx.set_magnetic_data(sta)
    mag = ctx.objective_and_gradient(x)[1]
    assert np.abs(grav + mag - joint).max() <= 64 * EPS * np.abs(joint).max()


def test_heavy_interpolation_sources():
    """Chain gather on a model whose control points drive thousands of rows (a
    CTA per source; the other chain tests' feed few): the gradient along a random
    step against a central difference of the objective (truncation and rounding
    below 1e-5 of the sum of magnitudes at a step of 1e-3 m)."""
    p = synth.voxel_contact_model(shape=(24, 24, 12), n_side=3, cp_stride=4)
    model = p.build_model()
    t = model.tables()
    fed = np.bincount(t["interp_src"], minlength=len(t["pos"]))
    assert fed.max() > 512
    ctx = p.make_context(model)
    ctx.set_gradient_gather(GATHER_CHAIN)
    ctx.set_collapsed_facets(COLLAPSED_DROP)
    ctx.set_scatter_stateless(True)
    rng = np.random.default_rng(1)
    x = model.assemble_parameters() + rng.normal(0.0, 3.0, model.n_dofs)
    g = ctx.objective_and_gradient(x)[1]
    step = rng.normal(0.0, 1.0, model.n_dofs)
    h = 1e-3
    fd = (ctx.objective(x + h * step) - ctx.objective(x - h * step)) / (2 * h)
    assert abs(fd - g @ step) <= 1e-5 * np.abs(g * step).sum()
