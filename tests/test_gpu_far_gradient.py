"""The FP32 far-field gradient kernel at the edges of its dispatch: far-field
ratios on both sides of 3 (series with and without the library fall-back),
one data type alone, station counts that leave a partial tile, several groups
and batched bodies.  Mixed gradient against the FP64 path's: 1e-5 of the
largest entry, the mixed path's stated gradient tolerance."""
import numpy as np
import pytest

from lithoinv3d_b200 import PREC_FP64, PREC_MIXED, synth

pytestmark = pytest.mark.gpu


def gradients(problem, tau, grav=True, mag=True):
    model = problem.build_model()
    x = model.assemble_parameters() + np.random.default_rng(2).normal(0.0, 3.0, model.n_dofs)
    ctx = problem.make_context(model)
    none = np.zeros((0, 3))
    if not grav:
        ctx.set_gravity_data(none)
    if not mag:
        ctx.set_magnetic_data(none)
    ctx.set_far_field_ratio(tau)
    out = []
    for p in (PREC_FP64, PREC_MIXED):
        ctx.set_precision(p)
        out.append(ctx.objective_and_gradient(x)[1])
    return out


@pytest.mark.parametrize("tau", [2.0, 2.99, 3.0, 4.0])
def test_ratios(tau):
    ref, got = gradients(synth.voxel_contact_model(shape=(9, 8, 5), n_side=17, n_groups=3, cp_stride=0, axis_scale=2.0), tau)
    assert np.abs(got - ref).max() <= 1e-5 * np.abs(ref).max()


@pytest.mark.parametrize("side", [1, 8, 9])
@pytest.mark.parametrize("data", ["gravity", "magnetic"])
def test_one_data_type(data, side):
    p = synth.icosphere_model(subdiv=2, n_side=side, spacing=37.0, freedom=synth.XYZ_FREE)
    ref, got = gradients(p, 3.0, grav=data == "gravity", mag=data == "magnetic")
    assert np.abs(got - ref).max() <= 1e-5 * np.abs(ref).max()


def test_batch():
    p = synth.batch_bodies_model(n_bodies=5, t_range=(60, 900), side_range=(3, 21), seed=4)
    ref, got = gradients(p, 3.0)
    assert np.abs(got - ref).max() <= 1e-5 * np.abs(ref).max()
