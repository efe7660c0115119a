"""A periodic lattice, and a batch, that fit the device with their rows one behind
the other and not with rows padded for the row tiles: they are created without
the padding, whichever of their arrays it is that does not fit."""
import pytest

pytestmark = pytest.mark.gpu


def descs(gpu, batch, prec, scale):
    shape = (67, 600, 1600 // scale) if not batch else (67, 160, 640 // scale)
    d = gpu.default_desc(nx=shape[0], ny=shape[1], nz=shape[2], mode=gpu.MODE_PHYSICS, precision=prec,
                         periodic=(1, 1, 1), tau=0.6)
    return [d] * (12 if batch else 1)


def make(gpu, batch, prec, scale=1):
    ds = descs(gpu, batch, prec, scale)
    return gpu.Batch(ds) if batch else gpu.Lattice(ds[0])


@pytest.mark.parametrize("batch", [False, True])
@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("part", [0.25, 0.75])
def test_created_without_padding(gpu, batch, prec, part):
    import torch
    small = make(gpu, batch, prec, 8)  # loads the kernels
    small.close()
    x = make(gpu, batch, prec)
    padded = x.info().device_bytes
    x.close()
    ds = descs(gpu, batch, prec, 1)
    nodes = sum(d.nx * d.ny * d.nz for d in ds)
    extra = nodes * 5 // 67 * 19 * (2 if prec else 4)  # 72 elements a row in place of 67
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    # room for the arrays, and for `part` of the padding
    filler = torch.empty(free - (padded - extra) - int(part * extra), dtype=torch.uint8, device="cuda")
    try:
        y = make(gpu, batch, prec)
    finally:
        del filler
        torch.cuda.empty_cache()
    assert abs((padded - y.info().device_bytes) / extra - 1) < 0.01
    if batch:
        assert y.lanes(1 << 20) == 0
    else:
        assert not y.streams_rows()
    y.close()
    # the padding alone decides: with room for it, it is there
    z = make(gpu, batch, prec)
    assert z.info().device_bytes == padded
    z.close()
