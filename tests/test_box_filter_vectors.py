"""The box filter's vector loads: the same factor on aligned fields and on
fields moved by one value (single loads) gives the same bits, on cubes and on
ragged grids; the FP64 oracle test covers the values."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape,factor", [((4, 4, 4), 4), ((20, 12, 8), 4), ((2, 6, 10), 2), ((34, 14, 6), 2),
                                          ((24, 16, 8), 8), ((18, 12, 6), 6), ((72, 24, 12), 12), ((9, 6, 3), 3)])
def test_aligned_and_shifted_fields_agree(gpu, shape, factor):
    import torch
    nx, ny, nz = shape
    n = nx * ny * nz
    g = torch.Generator(device="cuda").manual_seed(n)
    rho = 1 + 0.05 * torch.randn(n, generator=g, device="cuda")
    u = 0.05 * torch.randn(3 * n, generator=g, device="cuda")
    nc = n // factor ** 3
    got = []
    for shift in (0, 1):
        r, v = (torch.empty(a.numel() + 1, device="cuda") for a in (rho, u))
        r[shift:shift + n] = rho
        v[shift:shift + 3 * n] = u
        out = torch.empty(10 * nc, device="cuda")
        gpu.box_filter(r.data_ptr() + 4 * shift, v.data_ptr() + 4 * shift, shape, factor, out.data_ptr())
        torch.cuda.synchronize()
        got.append(out.cpu().numpy())
    assert np.array_equal(got[0], got[1])
    r64 = rho.double().cpu().numpy().reshape(nz // factor, factor, ny // factor, factor, nx // factor, factor)
    mean = r64.mean((1, 3, 5)).reshape(-1)
    assert np.max(np.abs(got[0][:nc] - mean)) <= 2e-7 * np.abs(mean).max()
