"""Pairs whose distances are zero or not numbers: the polynomial routes of the
FP64 and near-field kernels must leave them to the forms that test for them,
whatever the sign of the NaN that a zero distance produces."""
import numpy as np
import pytest

from lithoinv3d_b200 import GRAVITY, MAGNETIC, PREC_FP64, PREC_MIXED, synth
from lithoinv3d_b200.api import LithoError
from oracle_bindings import OracleModel

pytestmark = pytest.mark.gpu

# Long thin tetrahedron: from either end the other end's edges are short (their
# L / (d1 + d2) stays below 1/4), so only the zero distance itself can send the
# pair of a facet and a station on its vertex away from the polynomials.
V = np.array([[0.0, 0.0, -100.0], [400.0, 0.0, -100.0], [400.0, 60.0, -110.0], [380.0, 30.0, -160.0]])
F = np.array([[0, 2, 1], [0, 1, 3], [1, 2, 3], [0, 3, 2]], np.int32)


@pytest.mark.parametrize("precision", [PREC_FP64, PREC_MIXED])
@pytest.mark.parametrize("vertex", [0, 1, 2, 3])
@pytest.mark.parametrize("roll", [0, 1, 2])
def test_station_on_a_vertex(roll, vertex, precision):
    """A station on each vertex, as corner a, b and c of its facets: the forward
    is the oracle's (1e-6 of the largest entry, the mixed forward's tolerance;
    in mixed precision TMI on the vertex itself is finite only: it is singular
    there, and the facet frames round the zero distance to 1e-14 m, which the
    oracle's zero-distance branch does not see), Jacobian rows and the gradients
    of either data type and of both are finite (the oracle's difference quotients
    do not exist there; the second station's row is compared, 1e-6 of its largest
    entry as in the other Jacobian tests)."""
    sta = np.stack([V[vertex], V[vertex] + [700.0, -900.0, 800.0]])
    p = synth.Problem("long", [0.3], [0.02], [(V, np.roll(F, roll, axis=1).copy(), synth.XYZ_FREE)], sta, sta)
    model = p.build_model()
    ctx = p.make_context(model)
    ctx.set_precision(precision)
    x = model.assemble_parameters()
    om = OracleModel(model.tables(), p.densities, p.susceptibilities, p.inducing)
    om.scatter(x)
    gz, tmi = ctx.forward(x)
    assert np.isfinite(tmi).all()
    first = 0 if precision == PREC_FP64 else 1
    for got, want in ((gz, om.forward_gz(sta)), (tmi[first:], om.forward_tmi(sta)[first:])):
        assert np.abs(got - want).max() <= 1e-6 * np.abs(want).max()
    for which in (GRAVITY, MAGNETIC):
        J, Jt = ctx.jacobian(x, which), om.jacobian(sta[1:], 2 + which)[0]
        assert np.isfinite(J).all()
        assert np.abs(J[1] - Jt).max() <= 1e-6 * np.abs(Jt).max()
    none = np.zeros((0, 3))
    gradients = [ctx.objective_and_gradient(x)[1]]
    ctx.set_magnetic_data(none)
    gradients.append(ctx.objective_and_gradient(x)[1])
    ctx.set_gravity_data(none)
    ctx.set_magnetic_data(sta)
    gradients.append(ctx.objective_and_gradient(x)[1])
    assert all(np.isfinite(g).all() for g in gradients)


@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_overflowing_facet_is_not_dropped(sign):
    """A vertex so far away that the facet's area is inf - inf: the prediction
    is not a number and the objective is refused; the facet does not pass for
    one that contributes nothing."""
    sta = np.array([[10.0, 20.0, 1.0], [300.0, -40.0, 1.0]])
    p = synth.Problem("one facet", [0.3], [0.02], [(V[:3], F[:1], synth.XYZ_FREE)], sta, sta)
    model = p.build_model()
    ctx = p.make_context(model)
    x = model.assemble_parameters()
    x[:2] = sign * 1e200, 1e200
    gz, tmi = ctx.forward(x)
    assert not np.isfinite(gz).any() and not np.isfinite(tmi).any()
    with pytest.raises(LithoError):
        ctx.objective(x)
