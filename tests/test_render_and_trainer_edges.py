"""Edges of the raymarch's tiles and lane groups against the float32
restatement (bit for bit), and of the trainer's sample groups and blocks
against the FP64 gradient (1e-4 of its largest component, the bar of the other
batch sizes)."""
import numpy as np
import pytest

from oracle import closure_oracle as co
from oracle import render_oracle as ro

pytestmark = pytest.mark.gpu


# sizes around the 8 x 16 pixel tile, odd and single sample counts, extents that
# are powers of two and not, a camera inside the box, rays that saturate at once
@pytest.mark.parametrize("shape,size,steps,absorption", [((32, 16, 8), (1, 1), 1, 4.0), ((32, 16, 8), (9, 17), 3, 4.0),
                                                         ((20, 12, 9), (8, 16), 2, 0.0), ((20, 12, 9), (17, 15), 65, 50.0),
                                                         ((64, 3, 5), (33, 34), 127, 1.0)])
@pytest.mark.parametrize("f16", [True, False])
def test_render_tile_edges(gpu, shape, size, steps, absorption, f16):
    import torch
    rng = np.random.default_rng(steps)
    n = int(np.prod(shape))
    u = (0.05 * rng.standard_normal((3, n))).astype(np.float32)
    w, h = size
    for eye in ((-1.3 * shape[0], 1.7 * shape[1], 2.9 * shape[2]), (0.4 * shape[0], 0.6 * shape[1], 0.5 * shape[2])):
        m = gpu.camera(eye, (0.55 * shape[0], 0.5 * shape[1], 0.45 * shape[2]), aspect=w / h)
        p = gpu.velmag_params(inv_view_proj=m, camera_pos=eye, steps=steps, velmag_max=0.08, absorption=absorption,
                              round_f16=int(f16))
        d_u = torch.from_numpy(u).cuda()
        out = torch.full((h, w, 4), float("nan"), device="cuda")
        gpu.render_velmag(d_u.data_ptr(), shape, p, w, h, out.data_ptr())
        torch.cuda.synchronize()
        want = ro.render(u, shape, m, eye, w, h, steps=steps, vmax=0.08, absorption=absorption, round_f16=f16)
        assert np.array_equal(out.cpu().numpy(), want)


# one sample, one group and its neighbours, every block with one group (592), one
# more, and several groups a block with a ragged last one
@pytest.mark.parametrize("n", [1, 31, 32, 33, 592 * 32, 592 * 32 + 1, 50_001])
def test_gradient_group_edges(gpu, n):
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
