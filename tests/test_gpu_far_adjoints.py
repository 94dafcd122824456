"""The FP32 adjoints of the far-field gradient, formed beside the facet
constants: no launch of their own, and one block each for gravity and magnetic
stations that differ."""
import numpy as np
import pytest

from lithoinv3d_b200 import PREC_FP64, PREC_MIXED, synth

pytestmark = pytest.mark.gpu


def gradient(p, model, x, precision):
    """(gradient, launches of the evaluation beyond those of a forward)."""
    ctx = p.make_context(model)
    ctx.set_precision(precision)
    ctx.set_scatter_stateless(True)
    counts = []
    for call in (ctx.forward, ctx.objective_and_gradient):
        before = ctx.counters().launches
        out = call(x)
        counts.append(ctx.counters().launches - before)
    ctx.close()
    return out[1], counts[1] - counts[0]


def problem(grav, mag):
    p = synth.voxel_contact_model(shape=(8, 7, 5), n_groups=3, n_side=4)
    p.grav_xyz, p.mag_xyz = grav, mag
    return p


def test_no_launch_of_their_own():
    """Joint stations: the mixed gradient adds one kernel to the FP64 one's."""
    sta = synth.station_grid(9, 90.0, 1.0)
    p = problem(sta, sta)
    m = p.build_model()
    x = m.assemble_parameters()
    assert gradient(p, m, x, PREC_MIXED)[1] == gradient(p, m, x, PREC_FP64)[1] + 1


@pytest.mark.parametrize("n_grav,n_mag", [(1, 33), (127, 129), (300, 7), (0, 65), (65, 0)])
def test_station_sets_that_differ(n_grav, n_mag):
    """Mixed against FP64 gradient over three groups of different density and
    susceptibility, 1e-5 of the largest entry (the mixed gradient's tolerance)."""
    rng = np.random.default_rng(n_grav)
    sta = [np.column_stack([rng.uniform(-900.0, 900.0, (n, 2)), rng.uniform(1.0, 400.0, n)]) for n in (n_grav, n_mag)]
    p = problem(*sta)
    m = p.build_model()
    x = m.assemble_parameters()
    want = gradient(p, m, x, PREC_FP64)[0]
    assert np.abs(gradient(p, m, x, PREC_MIXED)[0] - want).max() <= 1e-5 * np.abs(want).max()
