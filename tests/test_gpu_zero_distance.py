"""Pairs whose distances are zero or not numbers: the polynomial routes of the
FP64 and near-field kernels must leave them to the forms that test for them,
whatever the sign of the NaN that a zero distance produces."""
import numpy as np
import pytest

from lithoinv3d_b200 import synth
from lithoinv3d_b200.api import LithoError

pytestmark = pytest.mark.gpu

V = np.array([[0.0, 0.0, -100.0], [400.0, 0.0, -100.0], [400.0, 60.0, -110.0], [380.0, 30.0, -160.0]])
F = np.array([[0, 2, 1], [0, 1, 3], [1, 2, 3], [0, 3, 2]], np.int32)


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
