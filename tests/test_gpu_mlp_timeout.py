"""A tcgen05 product that gives up on a wait ends queued training at its batch,
as it ends single steps.  The wait is made to run out by a limit of 0 polls
(every stage wait returns at once and the kernel drains its own work)."""
import numpy as np
import pytest

from test_gpu_mlp import Net

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("engine", [0, 2])
def test_train_rows_stops_at_the_batch(engine):
    """Five batches of a network whose first layer has ten K-blocks: the status
    is LF_ETIMEOUT and no loss after the first batch's is written.  With the
    limit restored a new network on that engine trains all five."""
    batch, n_in, n_out, batches = 128, 640, 70, 5
    g = torch.Generator(device="cuda").manual_seed(1)
    X = torch.randn((batch * batches, n_in), generator=g, device="cuda")
    Y = torch.randn((batch * batches, n_out), generator=g, device="cuda")
    rows = np.arange(batch * batches, dtype=np.int64)
    torch.cuda.synchronize()

    def train(net, losses):
        return net.lib.lf_mlp_train_rows(net.h, X.data_ptr(), Y.data_ptr(), len(rows), rows.ctypes.data, batches, 1e-3,
                                         losses.ctypes.data)

    net = Net(n_in, 128, 2, n_out, batch, seed=3)
    assert net.lib.lf_mlp_set_engine(net.h, engine) == 0
    losses = np.full(batches, -1.0, np.float32)
    try:
        assert net.lib.lf_set_device_wait_limit(0) == 0
        assert train(net, losses) == 5  # LF_ETIMEOUT
    finally:
        assert net.lib.lf_set_device_wait_limit(-1) == 0
    assert np.all(losses[1:] == -1.0)
    fresh = Net(n_in, 128, 2, n_out, batch, seed=3)
    assert fresh.lib.lf_mlp_set_engine(fresh.h, engine) == 0
    assert train(fresh, losses) == 0
    assert np.all(losses > 0.0)
