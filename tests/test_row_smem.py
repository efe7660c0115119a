"""One row-tile kernel serves fp32 lattices of five stages and of two: the
shared-memory limit of the kernel covers both, in any order."""
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

ROOT = Path(__file__).resolve().parents[1]


def test_limit_covers_every_lattice(tmp_path):
    sys.path.insert(0, str(ROOT / "gpu-sims_b200"))
    import build
    exe = tmp_path / "row_smem_check"
    subprocess.run([build.nvcc(), "-O1", "-std=c++17", "--expt-relaxed-constexpr", "-I", str(ROOT / "include"),
                    str(ROOT / "tests" / "row_smem_check.cu"), "-o", str(exe)] + build.ARCH, check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, env={**os.environ, "CUDA_VISIBLE_DEVICES": "-1"})
    assert r.returncode == 0, r.stdout


def lattice(gpu, shape, seed):
    rng = np.random.default_rng(seed)
    n = int(np.prod(shape))
    lat = gpu.Lattice(nx=shape[0], ny=shape[1], nz=shape[2], mode=gpu.MODE_PHYSICS, tau=0.6)
    lat.init_from_moments((1 + 0.01 * rng.standard_normal(n)).astype(np.float32),
                          (0.02 * rng.standard_normal((n, 3))).astype(np.float32))
    return lat


@pytest.mark.gpu
def test_deep_and_shallow_in_turn(gpu):
    """160 x 100 x 100 (five stages) and 101 x 97 x 64 (two), graphs and single
    launches in turn: the populations of each are those of the one-node kernel."""
    shapes = ((160, 100, 100), (101, 97, 64))
    want = []
    for i, s in enumerate(shapes):
        lat = lattice(gpu, s, i)
        lat.set_step_variant(1)
        lat.step(40)
        want.append(lat.read_populations_shifted())
        lat.close()
    lats = [lattice(gpu, s, i) for i, s in enumerate(shapes)]
    for k in (1, 18, 2, 19):
        for lat in lats:
            lat.step(k)
    for lat, w in zip(lats, want):
        lat.sync()
        assert np.array_equal(lat.read_populations_shifted(), w)
        lat.close()
