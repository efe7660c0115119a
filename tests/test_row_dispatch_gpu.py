"""Which kernel the automatic choice and graph mode take, so that the tests that
compare row tiles with another kernel do compare two kernels; and the forms of
the row tiles that those tests do not reach."""
import numpy as np
import pytest

from test_batch_lanes_gpu import initial
from test_row_tiles import CASES, test_matches_one_node_kernel as matches_one_node_kernel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [0, 1, 2])
def test_choice_by_grid_variant_and_closure(gpu, prec):
    for c in CASES.values():
        nx, ny, nz = c["shape"]
        lat = gpu.Lattice(nx=nx, ny=ny, nz=nz, mode=gpu.MODE_PHYSICS, precision=prec,
                          periodic=c.get("periodic", (0, 0, 0)), tau=0.57, smagorinsky_cs=c.get("cs", 0.0))
        assert lat.streams_rows(), c
        lat.set_step_variant(1)
        assert not lat.streams_rows()
        lat.close()
    lat = gpu.Lattice(nx=64, ny=64, nz=64, mode=gpu.MODE_PHYSICS, precision=prec, tau=0.6)
    assert not lat.streams_rows()
    lat.close()


SGS = {  # odd, ragged and whole rows with Smagorinsky
    "odd": dict(shape=(97, 60, 355), cs=0.1, trt=True, lid=True),
    "odd_periodic": dict(shape=(161, 51, 250), periodic=(1, 1, 1), cs=0.15, sphere=True),
    "ragged": dict(shape=(72, 80, 160), periodic=(0, 1, 0), cs=0.1, lid=True, sphere=True),
    "whole": dict(shape=(128, 120, 200), periodic=(1, 0, 0), cs=0.1, trt=True, sphere=True),
}


@pytest.mark.parametrize("prec,name", [(0, "odd"), (0, "odd_periodic"), (0, "ragged"), (1, "odd"), (1, "ragged"),
                                       (1, "whole"), (2, "odd_periodic")])
def test_smagorinsky(gpu, monkeypatch, prec, name):
    case = SGS[name]
    monkeypatch.setitem(CASES, "sgs", case)
    lat = gpu.Lattice(nx=case["shape"][0], ny=case["shape"][1], nz=case["shape"][2], mode=gpu.MODE_PHYSICS,
                      precision=prec, periodic=case.get("periodic", (0, 0, 0)), tau=0.57, smagorinsky_cs=case["cs"])
    assert lat.streams_rows()
    lat.set_params(smagorinsky_cs=0.0)  # the rule follows the parameters in effect
    assert lat.streams_rows()
    lat.close()
    matches_one_node_kernel(gpu, prec, "sgs")


def test_smagorinsky_changes_the_choice(gpu):
    """257 x 97 x 20 in fp16: row tiles without the term (0.8 of the row kernels'
    time), the row kernels with it (row tiles 1.3)."""
    lat = gpu.Lattice(nx=257, ny=97, nz=20, mode=gpu.MODE_PHYSICS, precision=1, periodic=(1, 0, 0), tau=0.57)
    assert lat.streams_rows()
    lat.set_params(smagorinsky_cs=0.1)
    assert not lat.streams_rows()
    lat.close()


@pytest.mark.parametrize("prec,shape", [(0, (512, 2, 2000)), (1, (512, 2, 2000)), (0, (129, 8000, 2)), (1, (129, 8000, 2)),
                                        (0, (67, 3, 4000)), (1, (67, 3, 4000)), (0, (95, 4000, 3))])
def test_thin_boxes_keep_the_row_kernels(gpu, prec, shape):
    lat = gpu.Lattice(nx=shape[0], ny=shape[1], nz=shape[2], mode=gpu.MODE_PHYSICS, precision=prec, tau=0.57)
    assert not lat.streams_rows()
    lat.close()


@pytest.mark.parametrize("case", [dict(shape=(160, 100, 100), lid=True, sphere=True),
                                  dict(shape=(161, 101, 101), periodic=(1, 0, 1), sphere=True, trt=True)])
def test_five_stage_fp32(gpu, monkeypatch, case):
    """fp32 above 120 MB without Smagorinsky: one block an SM, five stages."""
    monkeypatch.setitem(CASES, "deep", case)
    lat = gpu.Lattice(nx=case["shape"][0], ny=case["shape"][1], nz=case["shape"][2], mode=gpu.MODE_PHYSICS,
                      periodic=case.get("periodic", (0, 0, 0)), tau=0.57)
    assert lat.streams_rows()
    lat.close()
    matches_one_node_kernel(gpu, 0, "deep")


LANES = {  # shape, periodic: batches that graph mode runs in lanes
    "fp32": (0, [((64, 64, 64), (0, 0, 0)), ((101, 60, 50), (0, 0, 0)), ((96, 66, 60), (0, 1, 0)),
                 ((66, 64, 64), (1, 1, 1)), ((127, 40, 60), (0, 0, 1)), ((64, 48, 80), (0, 0, 0)),
                 ((128, 56, 50), (1, 0, 1))] * 2),
    # with a domain of the five-stage form beside two-stage ones
    "fp32_deep": (0, [((160, 100, 100), (0, 0, 0)), ((64, 64, 64), (0, 0, 0)), ((128, 56, 50), (1, 0, 1)),
                      ((96, 66, 60), (0, 1, 0)), ((66, 64, 64), (1, 1, 1)), ((127, 40, 60), (0, 0, 1)),
                      ((64, 48, 80), (0, 0, 0)), ((101, 60, 50), (0, 0, 0))]),
    "fp16": (1, [((96, 80, 40), (0, 0, 0)), ((71, 50, 40), (1, 0, 1)), ((33, 60, 70), (0, 0, 0)),
                 ((80, 80, 80), (0, 0, 1))] * 4),
}


@pytest.mark.parametrize("name", sorted(LANES))
def test_lanes_run_and_equal_single_domains(gpu, name):
    """Every domain bit for bit as advanced alone by the one-node kernel, over
    graphs from both parities and the launches after them."""
    prec, specs = LANES[name]
    wall = np.zeros((6, 3))
    wall[gpu.FACE_ZP] = (0.04, 0, 0)
    descs = [gpu.default_desc(nx=s[0], ny=s[1], nz=s[2], mode=gpu.MODE_PHYSICS, precision=prec,
                              periodic=per, tau=0.55 + 0.02 * i, wall_velocity=wall)
             for i, (s, per) in enumerate(specs)]
    b = gpu.Batch(descs)
    for i, d in enumerate(descs):
        mask, rho, u = initial(d, i)
        b.set_flags(i, mask)
        b.init_from_moments(i, rho, u)
    # the first graph is the tile kernel's, the next are the lanes' of either parity
    assert b.lanes(19) == 0 and b.lanes(16) == 0
    b.step(19)
    for steps in (403, 435):
        assert b.lanes(steps) > 0
        b.step(steps)
    assert b.lanes(17) > 0 and b.lanes(16) == 0  # their graphs exist now
    b.sync()
    for i, d in enumerate(descs):
        mask, rho, u = initial(d, i)
        lat = gpu.Lattice(d)
        lat.set_flags(mask)
        lat.init_from_moments(rho, u)
        lat.set_step_variant(1)
        lat.step(857)
        assert np.array_equal(b.read_populations(i), lat.read_populations()), i
        assert all(np.array_equal(x, y) for x, y in zip(b.read_moments(i), lat.read_moments())), i
        lat.close()
    b.close()
    b = gpu.Batch(descs)
    b.set_schedule(persistent=1)
    assert b.lanes(1000) == 0
    b.close()


@pytest.mark.parametrize("prec,shape,trt,cs,forced,plain", [
    (2, (77, 63, 81), True, 0.0, True, False), (1, (257, 80, 101), False, 0.1, True, False),
    (0, (149, 57, 46), True, 0.1, False, True), (0, (201, 48, 75), True, 0.1, True, False),
    (1, (88, 10, 400), False, 0.0, True, False), (0, (256, 10, 3000), False, 0.0, False, False)])
def test_a_force_on_one_node_rows_has_its_own_lines(gpu, prec, shape, trt, cs, forced, plain):
    """The one-node kernel rounds the half force differently, so the lines of
    forced rows that it would take (odd, ragged) are apart from the others', and
    those of the pair kernel are not: `forced` with a body force, `plain` without."""
    force, none = (1e-6, 0.0, 0.0), (0.0, 0.0, 0.0)
    for accel, want, other, want_other in ((force, forced, none, plain), (none, plain, force, forced)):
        lat = gpu.Lattice(nx=shape[0], ny=shape[1], nz=shape[2], mode=gpu.MODE_PHYSICS, precision=prec,
                          collision=gpu.COLL_TRT if trt else gpu.COLL_BGK, periodic=(1, 0, 1), tau=0.57,
                          smagorinsky_cs=cs, body_accel=accel)
        assert lat.streams_rows() == want
        lat.set_params(body_accel=other)
        assert lat.streams_rows() == want_other
        lat.close()
