"""Network.train on rows that are not flat: a vector of targets for one output,
images as inputs, non-contiguous views, fewer rows than a batch; and the shapes
it refuses."""
import numpy as np
import pytest

from lithoinv3d_b200.warmstart import Network

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def trained(X, Y, n_in, n_out):
    net = Network(n_in, n_out, width=128, depth=1, batch=128, seed=4)
    losses = net.train(X, Y, epochs=2, lr=1e-3, rng=np.random.default_rng(1))
    out = net.predict(torch.ones((3, n_in), device="cuda"))
    net.close()
    return losses, out


def test_row_shapes():
    g = torch.Generator(device="cuda").manual_seed(2)
    X = torch.randn((300, 24), generator=g, device="cuda")
    Y = torch.randn((300, 1), generator=g, device="cuda")
    want, out = trained(X, Y, 24, 1)
    for x, y in ((X, Y[:, 0]), (X.reshape(300, 4, 6), Y), (X.reshape(300, 2, 3, 4), Y[:, 0]),
                 (X.t().contiguous().t(), torch.cat([Y, Y]))):
        losses, o = trained(x, y, 24, 1)
        assert losses == want and torch.equal(o, out)
    one, o1 = trained(X[:, :1], Y, 1, 1)
    losses, o = trained(X[:, 0], Y, 1, 1)
    assert losses == one and torch.equal(o, o1)


def test_fewer_rows_than_a_batch():
    X, Y = torch.zeros((100, 24), device="cuda"), torch.zeros((100, 1), device="cuda")
    assert trained(X, Y, 24, 1)[0] == [0.0, 0.0]
    assert trained(X[:0], Y[:0], 24, 1)[0] == [0.0, 0.0]


@pytest.mark.parametrize("x,y", [((300, 23), (300, 1)), ((300, 25), (300, 1)), ((300, 24), (300, 2)), ((300, 24), (299, 1))])
def test_refused(x, y):
    with pytest.raises(IndexError):
        trained(torch.zeros(x, device="cuda"), torch.zeros(y, device="cuda"), 24, 1)
