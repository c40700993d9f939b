"""Which instances of a batch a thread-block cluster can go on with, on CPU
(cluster_solve.h through tests/native/cluster_fits_probe.cu): none on a size
that the device has no room for."""
from __future__ import annotations

import os
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
FULL = [148, 74, 36, 16, 7]  # clusters of 1, 2, 4, 8, 16 CTAs


@pytest.fixture(scope="module")
def smallest(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not Path(nvcc).exists():
        pytest.skip("nvcc not available")
    exe = tmp_path_factory.mktemp("fits") / "cluster_fits_probe"
    env = {k: v for k, v in os.environ.items() if k != "LD_PRELOAD"}
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17",
                    f"-I{ROOT / 'hpr-qp-c_b200' / 'csrc'}", "-o", str(exe),
                    str(ROOT / "tests" / "native" / "cluster_fits_probe.cu")], check=True, env=env)

    def run(n, m, warps, cap):
        text = " ".join(map(str, (n, m, warps, *cap)))
        return int(subprocess.run([str(exe)], input=text, capture_output=True, text=True, check=True, env=env).stdout)

    return run


# one CTA: 8 * (n + max(n, m) + m + 11 n + 5 m) bytes and 12 a row within 219 KB
@pytest.mark.parametrize("n,m,warps,want", [(1, 0, 20, 1), (640, 640, 20, 1), (1000, 500, 32, 1), (2000, 1000, 32, 2),
                                            (4000, 4000, 32, 8), (8190, 1000, 32, 16), (8190, 8190, 32, 0),
                                            (8191, 10, 32, 0), (10, 8191, 32, 0)])
def test_sizes(smallest, n, m, warps, want):
    assert smallest(n, m, warps, FULL) == want


@pytest.mark.parametrize("room", range(5))
def test_no_size_without_room(smallest, room):
    """Sizes from 1 to 2^room CTAs: an instance that needs a larger cluster
    stays where it is."""
    cap = [c if l <= room else 0 for l, c in enumerate(FULL)]
    for n, m in ((640, 640), (2000, 1000), (4000, 4000), (8190, 1000)):
        need = smallest(n, m, 32, FULL)
        assert smallest(n, m, 32, cap) == (need if need <= 1 << room else 0)
