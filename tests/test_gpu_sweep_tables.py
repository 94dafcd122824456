"""The side-by-side constraint sweep on tables that the model builder does not
make but lf_set_model_tables accepts, against a penalty evaluation at every
perturbed parameter vector (decisions and a fixed summation order: compared
exactly)."""
import numpy as np
import pytest

from lithoinv3d_b200 import Context, synth

pytestmark = pytest.mark.gpu


def context(V, F, dof_off, ref_vertex, ref_axis, ref_scale):
    """One group's raw tables in a stateless context."""
    ctx = Context()
    one, zero = np.array([0.3]), np.zeros(3)

    def d(a):
        return np.ascontiguousarray(a, np.float64).ctypes.data_as(ctx.lib.lf_set_model_tables.argtypes[2])

    def i(a):
        return np.ascontiguousarray(a, np.int32).ctypes.data_as(ctx.lib.lf_set_model_tables.argtypes[11])

    axis = np.ascontiguousarray(ref_axis, np.uint8)
    st = ctx.lib.lf_set_model_tables(ctx.h, 1, d(one), d(zero), d(zero), d(zero), d(zero), d(zero), len(V), d(V),
                                     len(F), i(F), i([0, len(F)]), len(dof_off) - 1, i(dof_off), i(ref_vertex),
                                     axis.ctypes.data_as(ctx.lib.lf_set_model_tables.argtypes[16]), d(ref_scale),
                                     None, None, None, 0, None, None)
    ctx._check(st, "set_model_tables")
    ctx.n_dofs, ctx.n_groups = len(dof_off) - 1, 1
    ctx.set_field(60.0, 10.0, 55000.0)
    ctx.set_gravity_data(np.array([[0.0, 0.0, 1.0]]))
    ctx.set_scatter_stateless(True)
    return ctx


def intervals(ctx, points):
    half = np.linspace(0.5, 9.0, len(points))
    ctx.set_constraints(points[:, :2], -points[:, 2] - half, -points[:, 2] + half, np.zeros(len(points)), weight=2.5)


def expected(ctx, x):
    g = np.zeros(len(x))
    for j in range(len(x)):
        p = x.copy()
        p[j] = x[j] + 1.0
        fp = ctx.constraint_penalty(p)
        p[j] = p[j] - 2.0
        g[j] = 2.5 * ((fp - ctx.constraint_penalty(p)) / 2.0)
    return g


def body():
    U, F = synth.icosphere(2)
    return U * 200.0 + [0.0, 0.0, -500.0], F


def test_parameter_that_writes_a_coordinate_twice():
    """z of every vertex twice, scaled by 0.5 and then by 1: the scatter's last
    write is the one that counts, on both sides of every step."""
    V, F = body()
    n = len(V)
    ctx = context(V, F, 2 * np.arange(n + 1), np.repeat(np.arange(n), 2), np.full(2 * n, 2), np.tile([0.5, 1.0], n))
    rng = np.random.default_rng(4)
    intervals(ctx, V[rng.integers(0, n, 50)] + rng.uniform(-0.6, 0.6, (50, 3)))
    x = V[:, 2].copy()
    want = expected(ctx, x)
    assert np.count_nonzero(want) > 0
    assert np.array_equal(ctx.constraint_gradient(x), want)


def test_two_parameters_on_one_coordinate():
    """Which of the two writes stays is the scatter's affair: such tables run
    pass by pass (at least a step and a scatter for each of the 2 np passes)."""
    V, F = body()
    n = len(V)
    vertex = np.concatenate([np.arange(n), [7]])
    ctx = context(V, F, np.arange(n + 2), vertex, np.full(n + 1, 2), np.ones(n + 1))
    intervals(ctx, V[:20] + 0.4)
    before = ctx.counters().launches
    ctx.constraint_gradient(V[vertex, 2])
    assert ctx.counters().launches - before >= 4 * (n + 1)


def test_lists_of_many_triangles():
    """1,024 fans whose hubs move together: the list's triangles times the points
    exceed 2^31, so that parameter is a whole pass; those numbered after it (a
    rim vertex, then a hub's neighbour) keep complete lists."""
    fans, rim, n = 1024, 1030, 2048
    assert fans * rim * n > 2 ** 31
    a = np.arange(rim) * (2 * np.pi / rim)
    one = np.concatenate([[[0.0, 0.0, 0.0]], np.stack([40.0 * np.cos(a), 40.0 * np.sin(a), np.full(rim, -30.0)], 1)])
    at = synth.station_grid(32, 100.0, -100.0)
    V = (at[:, None] + one[None]).reshape(-1, 3)
    k = np.arange(1, rim + 1)
    tri = np.stack([np.zeros_like(k), k, np.roll(k, -1)], 1)
    F = (np.arange(fans)[:, None, None] * (rim + 1) + tri[None]).reshape(-1, 3).astype(np.int32)
    hubs = np.arange(fans) * (rim + 1)
    moved = np.concatenate([hubs, [3], [4 * (rim + 1) + 7]])
    ctx = context(V, F, [0, fans, fans + 1, fans + 2], moved, np.full(fans + 2, 2), np.ones(fans + 2))
    rng = np.random.default_rng(1)
    t, u, f = rng.uniform(0, 2 * np.pi, n), rng.uniform(0.1, 0.9, n), rng.integers(0, fans, n)
    t[::4], u[::4], f[::4] = a[2] + 1e-4, 0.97, 0  # beside the other two parameters' vertices
    t[1::4], u[1::4], f[1::4] = a[6] - 1e-4, 0.97, 4
    pts = at[f] + np.stack([40.0 * u * np.cos(t), 40.0 * u * np.sin(t), -30.0 * u + rng.uniform(-0.4, 0.4, n)], 1)
    intervals(ctx, pts)
    x = V[moved[[0, fans, fans + 1]], 2]
    want = expected(ctx, x)
    assert np.all(want != 0)
    assert np.array_equal(ctx.constraint_gradient(x), want)


def launches(ctx, x):
    before = ctx.counters().launches
    g = ctx.constraint_gradient(x)
    return g, ctx.counters().launches - before


@pytest.mark.parametrize("numbers", [(64, 2048), (2048, 64, 2048)])
def test_route_of_few_long_lists(numbers):
    """16 parameters that each move up to 381 vertices: under few points side by
    side (fewer launches than passes), under many pass by pass (several launches
    each on the first, direct run), with the same values, in either order."""
    p = synth.voxel_contact_model(shape=(12, 10, 6), n_groups=2, n_side=4, cp_stride=4)
    m = p.build_model()
    rng = np.random.default_rng(7)
    x = m.assemble_parameters() + rng.normal(0.0, 3.0, m.n_dofs)
    ctx = p.make_context(m)
    ctx.set_scatter_stateless(True)
    ctx.forward(x)
    pos = ctx.positions(m.info().n_vertices)
    for n in numbers:
        mid = pos[rng.integers(0, len(pos), n)] + rng.uniform(-0.6, 0.6, (n, 3))
        half = rng.uniform(0.5, 9.0, n)
        ctx.set_constraints(mid[:, :2], -mid[:, 2] - half, -mid[:, 2] + half, rng.integers(0, 2, n), weight=2.5)
        want = expected(ctx, x)
        assert np.count_nonzero(want) > 0
        g, count = launches(ctx, x)
        assert np.array_equal(g, want)
        assert count < 2 * m.n_dofs if n == 64 else count >= 4 * 2 * m.n_dofs


def test_many_parameters_that_move_much():
    """70 parameters of 1,030 vertices each, which run as whole passes, do not
    hold back the 300 others: fewer launches than two per pass."""
    U, F = synth.icosphere(6)
    V = U * 200.0 + [0.0, 0.0, -500.0]
    heavy, each, light = 70, 1030, 300
    coordinate = np.arange(heavy * each)
    vertex = np.concatenate([coordinate % len(V), np.arange(light)])
    axis = np.concatenate([coordinate // len(V), np.full(light, 2)])
    off = np.concatenate([np.arange(heavy + 1) * each, heavy * each + np.arange(1, light + 1)])
    # a heavy parameter is a factor on its coordinates, so that one number writes them all
    scale = np.concatenate([V[vertex[:heavy * each], axis[:heavy * each]] / 1000.0, np.ones(light)])
    ctx = context(V, F, off, vertex, axis, scale)
    rng = np.random.default_rng(2)
    near = rng.integers(0, len(V), 64)
    near[::2] = rng.integers(0, light, 32)
    intervals(ctx, V[near] + rng.uniform(-0.3, 0.3, (64, 3)))
    x = np.concatenate([np.full(heavy, 1000.0), V[:light, 2]])
    want = expected(ctx, x)
    assert np.count_nonzero(want[:heavy]) > 0 and np.count_nonzero(want[heavy:]) > 0
    g, count = launches(ctx, x)
    assert np.array_equal(g, want)
    assert count < 2 * 2 * len(x)
