"""Tile choices and the fused update of the MLP kernels: the mma.sync GEMM's three tiles add an element's products
in the same order (equal bits), queued training equals single steps, and the update made with the gradients equals
Adam on the gradients that lf_mlp_gradients returns."""
import ctypes as C

import numpy as np
import pytest

from lithoinv3d_b200 import _native
from test_gpu_mlp import Net, rel

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def gemm(engine, a_t, b_t, A, B, M, N, K):
    lib = _native.load()
    a, b = (A.t().contiguous() if a_t else A), (B if b_t else B.t().contiguous())
    out = torch.zeros((M, N), device="cuda")
    torch.cuda.synchronize()
    st = lib.lf_gemm_bf16(engine, a_t, b_t, 0, M, N, K, C.c_void_p(a.data_ptr()), a.shape[1], C.c_void_p(b.data_ptr()),
                          b.shape[1], None, C.c_void_p(out.data_ptr()), N, None)
    assert st == 0
    return out


# M of 128, 4736 and 18944 rows by 128 columns: tiles of 32 (64 where K is no multiple of 64), 64 and 128
@pytest.mark.parametrize("a_t,b_t", [(0, 0), (0, 1), (1, 0), (1, 1)])
@pytest.mark.parametrize("K", [32, 64, 96, 512, 1056])
def test_gemm_tiles_give_the_same_sums(a_t, b_t, K):
    g = torch.Generator(device="cuda").manual_seed(K)
    A = torch.randn((18944, K), generator=g, device="cuda").bfloat16()
    B = torch.randn((128, K), generator=g, device="cuda").bfloat16()
    parts = [gemm(1, a_t, b_t, A[:m].contiguous(), B, m, 128, K) for m in (128, 4736, 18944)]
    assert torch.equal(parts[0], parts[2][:128]) and torch.equal(parts[1], parts[2][:4736])
    a, b = A[:4736].double(), B.double()
    # fp32 accumulation of K products, each addition off by at most 2^-22 (truncation in the tensor cores)
    assert bool(((parts[1].double() - a @ b.t()).abs() <= K * 2.0 ** -22 * (a.abs() @ b.abs().t())).all())


# either side of the tile count that sends a deep reduction to the TMA kernel
@pytest.mark.parametrize("M,N", [(128, 128), (512, 1408), (512, 1536)])
def test_auto_engine_deep_reduction(M, N):
    K = 2048
    g = torch.Generator(device="cuda").manual_seed(M + N)
    A, B = (torch.randn((n, K), generator=g, device="cuda").bfloat16() for n in (M, N))
    c, a, b = gemm(3, 0, 1, A, B, M, N, K).double(), A.double(), B.double()
    assert bool(((c - a @ b.t()).abs() <= K * 2.0 ** -22 * (a.abs() @ b.abs().t())).all())


# n_in 252: rows on 16-byte boundaries; 250 and 129: not, and ragged against the padding.  33 batches: one more than
# are queued at a time.  17 hidden layers: more than one launch of gradients holds.
@pytest.mark.parametrize("n_in,depth,batches", [(252, 2, 3), (250, 1, 33), (129, 17, 2)])
def test_train_rows_equals_single_steps(n_in, depth, batches):
    batch, n_out = 128, 70
    one, many = (Net(n_in, 128, depth, n_out, batch, seed=7) for _ in range(2))
    rng = np.random.default_rng(n_in)
    n = batch * batches + 5
    X = torch.tensor(rng.normal(size=(n, n_in)), dtype=torch.float32, device="cuda")
    Y = torch.tensor(rng.normal(size=(n, n_out)), dtype=torch.float32, device="cuda")
    rows = rng.permutation(n).astype(np.int64)
    losses, want = np.zeros(batches, np.float32), []
    for b in range(batches):
        idx = torch.as_tensor(rows[b * batch:(b + 1) * batch], device="cuda")
        x, y = X[idx].contiguous(), Y[idx].contiguous()
        torch.cuda.synchronize()
        loss = C.c_float()
        assert one.lib.lf_mlp_train_step(one.h, x.data_ptr(), y.data_ptr(), 1e-3, C.byref(loss)) == 0
        want.append(loss.value)
    args = (X.data_ptr(), Y.data_ptr(), n, rows.ctypes.data, batches, 1e-3, losses.ctypes.data)
    assert many.lib.lf_mlp_train_rows(many.h, *args) == 0
    assert np.array_equal(losses, np.array(want, np.float32))
    assert np.array_equal(one.params(), many.params())
    bad = rows.copy()
    bad[1] = n
    assert many.lib.lf_mlp_train_rows(many.h, args[0], args[1], n, bad.ctypes.data, *args[4:]) != 0
    assert np.array_equal(one.params(), many.params())


@pytest.mark.parametrize("engine", [0, 1, 3])
@pytest.mark.parametrize("n_in,depth", [(250, 2), (129, 17)])
def test_first_update_is_adam_on_the_gradients(engine, n_in, depth):
    batch, n_out, lr = 384, 70, 1e-3
    net = Net(n_in, 128, depth, n_out, batch, seed=9)
    assert net.lib.lf_mlp_set_engine(net.h, engine) == 0
    rng = np.random.default_rng(2)
    x, y = rng.normal(size=(batch, n_in)).astype(np.float32), rng.normal(size=(batch, n_out)).astype(np.float32)
    w0 = net.params().astype(np.float64)
    loss, g = net.gradients(x, y)
    dx, dy = torch.tensor(x, device="cuda"), torch.tensor(y, device="cuda")
    torch.cuda.synchronize()
    got = C.c_float()
    assert net.lib.lf_mlp_train_step(net.h, dx.data_ptr(), dy.data_ptr(), lr, C.byref(got)) == 0
    assert got.value == loss
    # the first step from zero moments: w - lr g / (|g| + eps).  1 - b1 and 1 - b2 carry fp32 rounding of b1 and b2
    # (2^-25 against 0.1 and 0.001: 3e-7 and 3e-5, half of the latter under the root), in c1 and c2 alike
    g = g.astype(np.float64)
    want = w0 - lr * g / (np.abs(g) + 1e-8)
    assert np.max(np.abs(net.params() - want)) <= lr * 5e-5 + 2.0 ** -23 * np.max(np.abs(w0))
    # the two ways of forming gradients (per layer, grouped) agree
    other = Net(n_in, 128, depth, n_out, batch, seed=9)
    assert other.lib.lf_mlp_set_engine(other.h, 1) == 0
    assert rel(g, other.gradients(x, y)[1].astype(np.float64)) < 2e-3
