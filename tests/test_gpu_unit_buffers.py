"""Buffers of the unit responses: the first column of a new context sizes them
for every other one, so no later column pays for an allocation."""
import numpy as np
import pytest

from lithoinv3d_b200 import synth
from lithoinv3d_b200.api import UNIT_GRAVITY, UNIT_INDUCED

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def context():
    p = synth.voxel_contact_model(shape=(16, 16, 8), n_groups=4, n_side=60)
    m = p.build_model()
    return p.make_context(m), m.assemble_parameters(), [len(f) for _, f, _ in p.meshes]


def test_first_column_sizes_the_buffers():
    """Free device memory stays where it is after the smallest group's first
    column, whatever the order of kinds (kernels are loaded by a first context)."""
    loaded, x, sizes = context()
    for kind in (UNIT_GRAVITY, UNIT_INDUCED):
        want = [loaded.unit_response(x, kind, g) for g in range(len(sizes))]
    order = np.argsort(sizes)
    for first, second in ((UNIT_GRAVITY, UNIT_INDUCED), (UNIT_INDUCED, UNIT_GRAVITY)):
        ctx, x, _ = context()
        ctx.unit_response(x, first, int(order[0]))
        free = torch.cuda.mem_get_info()[0]
        for kind in (first, second):
            got = {int(g): ctx.unit_response(x, kind, int(g)) for g in order}
            if kind == UNIT_INDUCED:
                assert all(np.array_equal(got[g], w) for g, w in enumerate(want))
        assert torch.cuda.mem_get_info()[0] == free
        ctx.close()
