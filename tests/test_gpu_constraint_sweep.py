"""The side-by-side constraint sweep of stateless contexts against the passes
it stands for: a penalty evaluation at every perturbed parameter vector, the
central differences of ConstraintHandler::gradient, and the positions of the
last pass left behind.  Classifications are decisions and the penalty is summed
in a fixed order, so everything is compared exactly."""
import numpy as np
import pytest

from lithoinv3d_b200 import synth

pytestmark = pytest.mark.gpu


def expected(ctx, x, weight):
    g = np.zeros(len(x))
    for j in range(len(x)):
        p = x.copy()
        p[j] = x[j] + 1.0
        fp = ctx.constraint_penalty(p)
        p[j] = p[j] - 2.0
        fm = ctx.constraint_penalty(p)
        g[j] = weight * ((fp - fm) / 2.0)
    return g


@pytest.mark.parametrize("stride,freedom,label,n", [(2, synth.Z_ONLY, False, 33), (2, synth.XYZ_FREE, True, 256),
                                                    (0, synth.Z_ONLY, False, 1), (3, synth.XYZ_FREE, False, 257)])
def test_sweep(stride, freedom, label, n):
    p = synth.voxel_contact_model(shape=(6, 5, 4), n_side=4, n_groups=3, cp_stride=stride, freedom_interior=freedom,
                                  seed=8, axis_scale=2.0)
    m = p.build_model()
    rng = np.random.default_rng(n)
    x = m.assemble_parameters() + rng.normal(0.0, 3.0, m.n_dofs)
    ctx = p.make_context(m)
    ctx.set_scatter_stateless(True)
    ctx.forward(x)
    pos = ctx.positions(m.info().n_vertices)
    mid = pos[rng.integers(0, len(pos), n)] + rng.uniform(-0.6, 0.6, (n, 3))  # classes that a step can flip
    half = rng.uniform(0.5, 9.0, n)
    ctx.set_constraints(mid[:, :2], -mid[:, 2] - half, -mid[:, 2] + half, rng.integers(0, 3, n), weight=2.5)
    if label:
        lab = np.ascontiguousarray(p.extra["labels"].transpose(2, 1, 0)[::-1], np.int32)
        lab[:, ::2, :] = -1
        ctx.set_label_grid(lab, (-300.0, -250.0, -400.0), (100.0, 100.0, 100.0))
        ctx.set_bottom_depth(-390.0)
    want = expected(ctx, x, 2.5)
    left = ctx.positions(len(pos))
    for _ in range(2):
        assert np.array_equal(ctx.constraint_gradient(x), want)
        assert np.array_equal(ctx.positions(len(pos)), left)
    assert n < 33 or np.count_nonzero(want) > 0


def test_parameter_that_moves_a_whole_mesh():
    """Control points so sparse that some drive thousands of vertices: those
    parameters run as whole passes beside the others."""
    p = synth.voxel_contact_model(n_side=4)
    m = p.build_model()
    t = m.tables()
    rows = np.bincount(t["interp_src"], minlength=len(t["pos"]))
    per_dof = np.add.reduceat(rows[t["ref_vertex"]], t["dof_off"][:-1])
    assert per_dof.max() > 1024
    rng = np.random.default_rng(5)
    x = m.assemble_parameters() + rng.normal(0.0, 3.0, m.n_dofs)
    ctx = p.make_context(m)
    ctx.set_scatter_stateless(True)
    ctx.forward(x)
    pos = ctx.positions(len(t["pos"]))
    mid = pos[rng.integers(0, len(pos), 40)] + rng.uniform(-0.6, 0.6, (40, 3))
    half = rng.uniform(0.5, 9.0, 40)
    ctx.set_constraints(mid[:, :2], -mid[:, 2] - half, -mid[:, 2] + half, rng.integers(0, 4, 40), weight=2.5)
    want = expected(ctx, x, 2.5)
    assert np.array_equal(ctx.constraint_gradient(x), want)
