"""Training pass of the learned start over batch sizes (sample tiles of 32 and 64 with remainders,
one and many gradient slices) against the numpy network in FP64.

FP32 rounding: products of 128 terms and sums over at most a few hundred samples in a row before
the partial sums are added, so each gradient entry is within about 300 x 6e-8 of the sum of its
terms' sizes; 2e-5 of the largest entry is asked for, and 1e-5 of the outputs' scale."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 17, 32, 33, 64, 65, 753, 4864, 4865, 8192, 20001])
def test_loss_grad_and_forward(ccx, n):
    mlp = pytest.importorskip("mlp")
    r = np.random.RandomState(n)
    m = ccx.Learner()
    p = np.concatenate([0.3 * r.uniform(-1, 1, k) if k > 1 else r.uniform(-1, 1, k)
                        for k in (18 * 128, 128, 128 * 128, 128, 128 * 128, 128, 128, 1)]).astype(np.float32)
    m.set_params(p)
    X = r.standard_normal((n, 18)).astype(np.float32)
    y = r.standard_normal(n).astype(np.float32)
    loss, grad = m.loss_grad(X, y)
    want_loss, want = mlp.loss_grad(p, X, y)
    assert abs(loss - want_loss) <= 1e-5 * want_loss
    assert np.abs(grad - want).max() <= 2e-5 * np.abs(want).max()
    out, _ = mlp.forward(p, X)
    assert np.abs(m.infer(X, tensor_cores=False) - out).max() <= 1e-5 * max(np.abs(out).max(), 1.0)
    # a smaller batch afterwards, through the same workspaces
    l2, g2 = m.loss_grad(X[: max(1, n // 3)], y[: max(1, n // 3)])
    w2, want2 = mlp.loss_grad(p, X[: max(1, n // 3)], y[: max(1, n // 3)])
    assert abs(l2 - w2) <= 1e-5 * w2 and np.abs(g2 - want2).max() <= 2e-5 * np.abs(want2).max()
