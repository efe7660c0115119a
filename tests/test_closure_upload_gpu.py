"""Installing a network keeps its operands in memory the lattice has: no
allocation, and the next steps use the new network."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_closure_allocates_nothing(gpu):
    from oracle import closure_oracle as co
    lat = gpu.Lattice(nx=32, ny=16, nz=16, mode=gpu.MODE_PHYSICS, periodic=(1, 1, 1), tau=0.52, smagorinsky_cs=0.15)
    before = lat.info().device_bytes
    lat.set_closure(co.random_net(11))
    assert lat.info().device_bytes == before
    lat.close()


def test_networks_in_turn(gpu):
    """Two networks installed one after the other, without a wait between: each
    step equals a fresh lattice's with that network."""
    from oracle import closure_oracle as co
    shape = (40, 20, 12)
    n = int(np.prod(shape))
    u = (0.02 * np.random.default_rng(1).standard_normal((n, 3))).astype(np.float32)
    nets = [co.random_net(s, mean=np.array([0, 0, 0, 0, 0, 0, -6.0, 0, 0]),
                          iscale=np.array([1, 1, 1, 1, 1, 1, 0.5, 1, 50.0])) for s in (1, 2)]

    def lattice():
        lat = gpu.Lattice(nx=shape[0], ny=shape[1], nz=shape[2], mode=gpu.MODE_PHYSICS, periodic=(1, 1, 1), tau=0.52,
                          smagorinsky_cs=0.15)
        lat.init_from_moments(np.ones(n, np.float32), u)
        return lat

    got = lattice()
    for net in nets * 2:
        got.set_closure(net)
        got.step(18)
    want = lattice()
    for net in nets * 2:
        want.set_closure(None)
        want.set_closure(net)
        want.sync()
        want.step(18)
        want.sync()
    assert np.array_equal(got.read_populations_shifted(), want.read_populations_shifted())
    got.close()
    want.close()
