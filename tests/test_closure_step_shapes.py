"""The closure step's network on warp-level matrix products, at the shapes
where a warp is only partly filled: against the FP64 oracle, at the bar of the
full-warp tests (3e-5 of the velocity scale for fp32 storage)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", [0, 1])
@pytest.mark.parametrize("shape,open_x", [((33, 10, 9), False), ((66, 9, 7), False), ((96, 5, 6), False),
                                          ((5, 7, 6), False), ((40, 9, 8), True)])
def test_closure_step_matches_fp64(gpu, oracle, shape, open_x, variant):
    from oracle import closure_oracle as co
    net = co.random_net(11, mean=np.array([0, 0, 0, 0, 0, 0, -6.0, 0, 0]),
                        iscale=np.array([1, 1, 1, 1, 1, 1, 0.5, 1, 50.0]))
    nx, ny, nz = shape
    n = nx * ny * nz
    rng = np.random.default_rng(5)
    u = (0.02 * rng.standard_normal((3, n))).astype(np.float32)
    kw = dict(periodic=(0, 1, 1) if open_x else (1, 1, 1))
    wall = np.zeros((6, 3))
    if open_x:
        wall[gpu.FACE_XM] = (0.02, 0.0, 0.0)
        kw.update(open_x=(gpu.OPEN_VELOCITY, gpu.OPEN_PRESSURE), open_rho=(0.0, 1.0))
    lat = gpu.Lattice(nx=nx, ny=ny, nz=nz, mode=gpu.MODE_PHYSICS, tau=0.52, smagorinsky_cs=0.15,
                      wall_velocity=wall, **kw)
    lat.set_closure(net)
    lat.init_from_moments(np.ones(n, np.float32), np.ascontiguousarray(u.T))
    lat.set_step_variant(variant)
    lat.step(20)
    lat.sync()
    _, got = lat.read_moments()
    st = oracle.ExtState(shape, tau=0.52, smag_cs=0.15, wall=wall, net=net, **kw)
    st.init(np.ones(n), u.astype(np.float64))
    st.step(20)
    assert np.max(np.abs(got.T - st.u)) <= 3e-5 * np.abs(st.u).max()
    lat.close()
