"""The autotuner and the lanes of graph mode: it times them, a cache line that was
measured without them does not stand in for that, and a chosen schedule comes
back from the cache with its mode."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

ROOT = Path(__file__).resolve().parents[1]
PROGRAM = """
import sys
sys.path.insert(0, "gpu-sims_b200")
import lbm
descs = [lbm.default_desc(nx=64, ny=64, nz=64, mode=lbm.MODE_PHYSICS, precision=1, tau=0.6)] * 32
b = lbm.Batch(descs)
b.init_equilibrium()
s = b.autotune(10)
print(s.rows_per_block, s.z_per_thread, s.persistent, b.lanes(17))
"""


def tuned(cache):
    r = subprocess.run([sys.executable, "-c", PROGRAM], capture_output=True, text=True, cwd=ROOT,
                       env={**os.environ, "LBM_AUTOTUNE_CACHE": str(cache)})
    assert r.returncode == 0, r.stderr
    return [int(v) for v in r.stdout.split()]


def test_lanes_are_timed_and_cached(gpu, tmp_path):
    """32 cavities of 64^3 in fp16: lanes take 0.6 of the tile kernel's time and of
    persistent mode's."""
    cache = tmp_path / "cache"
    # precision, collision, log2 nodes, log2 domains, rows, z, persistent: before lanes
    cache.write_text("1 0 23 5 4 4 1\n")
    first = tuned(cache)
    assert first[2] == 0 and first[3] > 0  # their graph is the timed one: no wait for it to pay
    lines = cache.read_text().splitlines()
    assert lines[0] == "1 0 23 5 4 4 1" and len(lines) == 2
    second = tuned(cache)  # from the cache: nothing is measured or added
    assert second[:3] == first[:3] and len(cache.read_text().splitlines()) == 2
