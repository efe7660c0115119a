"""Rows of periodic lattices are padded for the row tiles where those run, and
nowhere else: the population memory of the others is that of their nodes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def slot_elements(make):
    """Elements of a slot array, from the memory that only the populations' width changes."""
    sizes = []
    for prec in (0, 1):
        x = make(prec)
        sizes.append(x.info().device_bytes)
        x.close()
    return (sizes[0] - sizes[1]) // 38


@pytest.mark.parametrize("shape,row", [((2, 300, 60), 2), ((9, 30, 41), 9), ((33, 10, 12), 33), ((65, 64, 64), 65),
                                       ((67, 30, 280), 72), ((1001, 20, 20), 1001)])
def test_lattice_rows(gpu, shape, row):
    nx, ny, nz = shape
    got = slot_elements(lambda prec: gpu.Lattice(nx=nx, ny=ny, nz=nz, mode=gpu.MODE_PHYSICS, precision=prec,
                                                 periodic=(1, 1, 1), tau=0.6))
    assert got == -(-row * ny * nz // 64) * 64


def test_batch_rows(gpu):
    """Domains too few for lanes."""
    def batch(prec):
        return gpu.Batch([gpu.default_desc(nx=9, ny=16, nz=32, mode=gpu.MODE_PHYSICS, precision=prec,
                                           periodic=(1, 1, 1), tau=0.6)] * 2)
    b = batch(0)
    assert b.lanes(1 << 20) == 0
    b.close()
    assert slot_elements(batch) == 2 * 9 * 16 * 32


@pytest.mark.parametrize("shape", [(9, 30, 41), (67, 30, 280)])
def test_set_params_keeps_the_layout(gpu, shape):
    n = int(np.prod(shape))
    rng = np.random.default_rng(2)
    rho = (1 + 0.01 * rng.standard_normal(n)).astype(np.float32)
    u = (0.02 * rng.standard_normal((n, 3))).astype(np.float32)
    got = []
    for change in (False, True):
        lat = gpu.Lattice(nx=shape[0], ny=shape[1], nz=shape[2], mode=gpu.MODE_PHYSICS, periodic=(1, 0, 1), tau=0.6)
        lat.init_from_moments(rho, u)
        lat.step(3)
        if change:
            lat.set_params(tau=0.6)
        lat.step(20)
        lat.sync()
        got.append(lat.read_populations_shifted())
        lat.close()
    assert np.array_equal(*got)
