"""The row-tile step (gpu-sims_b200/csrc/phys_rows.cuh): its index arithmetic
against the node formulas on the CPU, and on the GPU the automatic choice
against the one-node kernel, bit for bit."""
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]


def test_index_arithmetic(tmp_path):
    """Every element read and written, over periodic and walled axes, odd and
    even rows, one row per tile to sixteen, both element sizes."""
    sys.path.insert(0, str(ROOT / "gpu-sims_b200"))
    import build
    exe = tmp_path / "row_tiles_check"
    subprocess.run([build.nvcc(), "-O1", "-std=c++17", "--expt-relaxed-constexpr", "-I", str(ROOT / "include"),
                    str(ROOT / "tests" / "row_tiles_check.cu"), "-o", str(exe)] + build.ARCH, check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout


# Grids that the automatic choice gives to row tiles: odd and even rows, the
# longest and the shortest row, tiles of one row, of several and with a ragged
# last one, every periodic axis, all features.
CASES = {
    "walls_odd": dict(shape=(67, 30, 280), lid=True, sphere=True),
    "periodic_x": dict(shape=(71, 23, 360), periodic=(1, 0, 0), sphere=True, trt=True),
    "periodic_yz": dict(shape=(82, 37, 180), periodic=(0, 1, 1), sphere=True),
    "periodic": dict(shape=(161, 17, 180), periodic=(1, 1, 1), cs=0.15, sphere=True),
    "smag_trt": dict(shape=(81, 29, 210), cs=0.1, trt=True, lid=True),
    "force": dict(shape=(437, 11, 101), periodic=(1, 0, 0), force=True, sphere=True),
    "open": dict(shape=(95, 25, 220), open_x=True, sphere=True),
    "longest_row": dict(shape=(511, 6, 180), lid=True),
    "short_row": dict(shape=(66, 33, 220), periodic=(1, 0, 1)),
}


@pytest.mark.gpu
@pytest.mark.parametrize("prec", [0, 1, 2])
@pytest.mark.parametrize("case", sorted(CASES))
def test_matches_one_node_kernel(gpu, prec, case):
    """Populations and moments equal the one-node kernel's bit for bit: the
    collision is the same fused operations in both.  With a body force the bar
    is that of the other kernel variants, a few units in the last place."""
    c = CASES[case]
    nx, ny, nz = c["shape"]
    n = nx * ny * nz
    wall = np.zeros((6, 3))
    if c.get("lid"):
        wall[gpu.FACE_ZP] = (0.05, 0.01, 0.0)
        wall[gpu.FACE_XM] = (0.0, 0.02, 0.0)
    kw = {}
    if c.get("open_x"):
        wall[gpu.FACE_XM] = (0.03, 0.0, 0.0)
        kw.update(open_x=(gpu.OPEN_VELOCITY, gpu.OPEN_PRESSURE), open_rho=(0.0, 1.0))
    if c.get("force"):
        kw["body_accel"] = (1e-5, -2e-6, 3e-6)
    rng = np.random.default_rng(3)
    u = (0.02 * rng.standard_normal((n, 3))).astype(np.float32)
    rho = (1.0 + 0.01 * rng.standard_normal(n)).astype(np.float32)
    got = []
    for variant in (0, 1):
        lat = gpu.Lattice(nx=nx, ny=ny, nz=nz, mode=gpu.MODE_PHYSICS, precision=prec,
                          collision=gpu.COLL_TRT if c.get("trt") else gpu.COLL_BGK,
                          periodic=c.get("periodic", (0, 0, 0)), tau=0.57, smagorinsky_cs=c.get("cs", 0.0),
                          wall_velocity=wall, **kw)
        if c.get("sphere"):
            z, y, x = np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")
            m = (x - nx // 2) ** 2 + (y - ny // 3) ** 2 + (z - nz // 2) ** 2 <= max(2, ny // 5) ** 2
            m[nz // 4, ny // 2:, :] = True  # and a wall that meets the faces
            lat.set_flags(m.astype(np.uint8))
        lat.init_from_moments(rho, u)
        lat.set_step_variant(variant)
        lat.step(7)   # both parities, single launches
        lat.step(18)  # a graph of 16 and the launch that writes the moments
        lat.sync()
        got.append((lat.read_populations_shifted(), *lat.read_moments()))
        lat.close()
    for a, b in zip(*got):
        if c.get("force"):
            assert np.max(np.abs(a - b)) <= {0: 1e-4, 1: 1e-3, 2: 1e-2}[prec] * np.abs(b).max()
        else:
            assert np.array_equal(a, b)
