"""A row-streaming step whose bounded wait runs out: the protocol that lands its
copies, on the CPU, and on the GPU the error status and the recovery (the wait
has no polls, so that it gives up at once: nothing faults)."""
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]


def test_drain_protocol(tmp_path):
    sys.path.insert(0, str(ROOT / "gpu-sims_b200"))
    import build
    exe = tmp_path / "row_drain_check"
    subprocess.run([build.nvcc(), "-O1", "-std=c++17", "--expt-relaxed-constexpr", "-I", str(ROOT / "include"),
                    str(ROOT / "tests" / "row_drain_check.cu"), "-o", str(exe)] + build.ARCH, check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


def moments(shape, seed):
    rng = np.random.default_rng(seed)
    n = int(np.prod(shape))
    return (1 + 0.01 * rng.standard_normal(n)).astype(np.float32), (0.02 * rng.standard_normal((n, 3))).astype(np.float32)


# two blocks an SM with two and with five stages, one block with five, no periodic axis and all
@pytest.mark.gpu
@pytest.mark.parametrize("prec,shape,per,cs", [(0, (101, 97, 64), (0, 0, 0), 0.0), (1, (97, 80, 80), (1, 1, 1), 0.0),
                                               (2, (161, 60, 80), (0, 1, 0), 0.1), (0, (160, 100, 100), (1, 0, 0), 0.0)])
def test_step_gives_up_and_recovers(gpu, prec, shape, per, cs):
    def lattice():
        lat = gpu.Lattice(nx=shape[0], ny=shape[1], nz=shape[2], mode=gpu.MODE_PHYSICS, precision=prec, periodic=per,
                          tau=0.6, smagorinsky_cs=cs)
        assert lat.streams_rows()
        lat.init_from_moments(*moments(shape, 1))
        return lat

    fresh = lattice()
    fresh.step(20)
    want = fresh.read_populations_shifted()
    fresh.close()
    lat = lattice()
    lat.set_row_wait_limit(0)
    lat.step(20)  # a graph of 16 and four single launches, each of which gives up
    with pytest.raises(gpu.LbmError) as e:
        lat.sync()
    assert e.value.code == gpu.ERR_TIMEOUT
    with pytest.raises(gpu.LbmError) as e:
        lat.step(1)  # the state is not whole: it needs an init first
    assert e.value.code == gpu.ERR_STATE
    lat.set_row_wait_limit(-1)
    lat.init_from_moments(*moments(shape, 1))
    lat.step(20)
    lat.sync()
    assert np.array_equal(lat.read_populations_shifted(), want)
    lat.close()


@pytest.mark.gpu
def test_lanes_give_up_and_recover(gpu):
    shape = (96, 80, 40)
    descs = [gpu.default_desc(nx=shape[0], ny=shape[1], nz=shape[2], mode=gpu.MODE_PHYSICS, precision=1, tau=0.6)] * 16
    b = gpu.Batch(descs)
    got = []
    for limit in (-1, 0, -1):
        for i in range(len(descs)):
            b.init_from_moments(i, *moments(shape, i))
        b.set_row_wait_limit(limit)
        assert b.lanes(400) > 0
        b.step(400)  # graphs of lanes; the last sixteen steps are the tile kernel's
        if limit == 0:
            with pytest.raises(gpu.LbmError) as e:
                b.sync()
            assert e.value.code == gpu.ERR_TIMEOUT
            with pytest.raises(gpu.LbmError) as e:
                b.step(1)
            assert e.value.code == gpu.ERR_STATE
        else:
            b.sync()
            got.append([b.read_populations(i) for i in range(len(descs))])
    assert all(np.array_equal(x, y) for x, y in zip(*got))
    b.close()
