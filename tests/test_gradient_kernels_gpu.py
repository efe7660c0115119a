"""The gradient kernels of small and large batches against the FP64 gradient (1e-4
of its largest component, the bar of the other batch sizes)."""
import numpy as np
import pytest

from oracle import closure_oracle as co

pytestmark = pytest.mark.gpu


# around the size where the kernel changes, and one whole round of its blocks
@pytest.mark.parametrize("n", [24_575, 24_576, 24_577, 296 * 128, 296 * 128 + 1])
def test_gradient_kernels(gpu, n):
    import torch
    rng = np.random.default_rng(n)
    X = rng.standard_normal((n, 9)).astype(np.float32)
    X[:, 6] = -6 + 2 * X[:, 6]
    t = rng.uniform(0, 3, n).astype(np.float32)
    w = rng.uniform(0.1, 2, n).astype(np.float32)
    net = co.random_net(4, mean=np.array([0, 0, 0, 0, 0, 0, -6.0, 0, 0]),
                        iscale=np.array([1, 1, 1, 1, 1, 1, 0.5, 1, 1.0]))
    tr = gpu.Trainer(net)
    dX, dt, dw = (torch.from_numpy(a).cuda() for a in (X, t, w))
    ws = float(1.0 / w.astype(np.float64).sum())
    g, loss = tr.grad(dX.data_ptr(), dt.data_ptr(), dw.data_ptr(), n, ws)
    g2, loss2 = tr.grad(dX.data_ptr(), dt.data_ptr(), dw.data_ptr(), n, ws)
    tr.close()
    L, gw = co.loss_and_grad(co.kernel_net(net), X.astype(np.float64), t, w, np.float32(ws))
    assert abs(loss - L) <= 1e-5 * L
    assert np.max(np.abs(g - gw)) <= 1e-4 * np.abs(gw).max()
    assert np.array_equal(g, g2) and loss == loss2
