"""Batches large enough that graph mode runs lanes of row-tile steps: every
domain equals the same domain advanced alone, bit for bit, over graphs, the
launches after them and both starting parities; a batch in persistent mode and
one of the same domains by the tile kernel alone agree too."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SPECS = [  # shape, periodic, tau, lid: sixteen domains, 2.9 million nodes, rows of 16 to 140
    ((96, 80, 40), (0, 0, 0), 0.6, 0.05), ((64, 64, 64), (0, 0, 0), 0.55, 0.03), ((71, 50, 40), (1, 0, 1), 0.7, 0.0),
    ((140, 40, 30), (0, 1, 0), 0.52, 0.04), ((33, 60, 70), (0, 0, 0), 0.8, 0.02), ((48, 48, 48), (1, 1, 1), 0.6, 0.0),
    ((80, 80, 30), (0, 0, 1), 0.57, 0.0), ((16, 90, 90), (0, 0, 0), 0.6, 0.05)] * 2


def initial(d, seed):
    n = d.nx * d.ny * d.nz
    rng = np.random.default_rng(seed)
    return ((rng.random(n) < 0.02).astype(np.uint8), (1 + 0.005 * rng.standard_normal(n)).astype(np.float32),
            (0.01 * rng.standard_normal((n, 3))).astype(np.float32))


@pytest.mark.parametrize("prec,coll", [(0, 0), (1, 1), (2, 1)])
def test_lanes_equal_single_domains(gpu, prec, coll):
    descs = []
    for shape, per, tau, lid in SPECS:
        wall = np.zeros((6, 3))
        wall[gpu.FACE_ZP] = (lid, 0, 0)
        descs.append(gpu.default_desc(nx=shape[0], ny=shape[1], nz=shape[2], mode=gpu.MODE_PHYSICS, precision=prec,
                                      collision=coll, periodic=per, tau=tau, wall_velocity=wall))
    want = []
    for i, d in enumerate(descs):
        mask, rho, u = initial(d, i)
        lat = gpu.Lattice(d)
        lat.set_flags(mask)
        lat.init_from_moments(rho, u)
        lat.set_step_variant(1)
        lat.step(54)
        want.append((lat.read_populations(), *lat.read_moments()))
        lat.close()
    for persistent in (0, 1):
        b = gpu.Batch(descs)
        for i, d in enumerate(descs):
            mask, rho, u = initial(d, i)
            b.set_flags(i, mask)
            b.init_from_moments(i, rho, u)
        b.set_schedule(rows_per_block=4, z_per_thread=8, persistent=persistent)
        b.step(19)  # one graph and three launches: the next graph starts from the other parity
        b.step(35)
        b.sync()
        for i in range(len(descs)):
            got = (b.read_populations(i), *b.read_moments(i))
            assert all(np.array_equal(x, y) for x, y in zip(got, want[i])), (persistent, i)
        b.close()
