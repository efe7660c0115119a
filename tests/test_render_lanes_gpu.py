"""One or two lanes a ray of the raymarch, by steps and pixels: both bit for bit
the float32 restatement's image."""
import numpy as np
import pytest

from oracle import render_oracle as ro

pytestmark = pytest.mark.gpu


# one lane: fewer than 24 steps on 148 x 1,024 pixels and more, fewer than 4 on less; partial
# tiles of 8 x 32 pixels; blocks that no ray of theirs enters the volume from
@pytest.mark.parametrize("size,steps", [((8, 32), 3), ((9, 33), 2), ((9, 33), 4), ((148, 1024), 5), ((148, 1023), 5),
                                        ((1025, 149), 23), ((1025, 149), 24)])
@pytest.mark.parametrize("f16", [True, False])
def test_render_lanes(gpu, size, steps, f16):
    import torch
    shape = (20, 16, 9)
    rng = np.random.default_rng(steps)
    u = (0.05 * rng.standard_normal((3, int(np.prod(shape))))).astype(np.float32)
    w, h = size
    eye = (-30.0, 25.0, 40.0)
    m = gpu.camera(eye, (16.0, 8.0, 4.0), aspect=w / h)
    p = gpu.velmag_params(inv_view_proj=m, camera_pos=eye, steps=steps, velmag_max=0.08, round_f16=int(f16))
    d_u = torch.from_numpy(u).cuda()
    out = torch.full((h, w, 4), float("nan"), device="cuda")
    gpu.render_velmag(d_u.data_ptr(), shape, p, w, h, out.data_ptr())
    torch.cuda.synchronize()
    want = ro.render(u, shape, m, eye, w, h, steps=steps, vmax=0.08, round_f16=f16)
    got = out.cpu().numpy()
    assert np.array_equal(got, want)
    assert (got[..., 3] > 0).any() and (got[..., 3] == 0).any()
