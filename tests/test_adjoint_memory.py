"""What nb_adj_forward keeps, and how much memory that takes."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
REPO = os.path.dirname(HERE)
GIB = 1 << 30


@pytest.fixture(scope="module")
def fits(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    out = str(tmp_path_factory.mktemp("tape") / "adj_tape_probe")
    subprocess.run([nvcc, "-O1", "-std=c++17", "-I", os.path.join(REPO, "include"), "-I",
                    os.path.join(REPO, "utc_gb300", "csrc"), os.path.join(HERE, "adj_tape_probe.cu"), "-o", out],
                   check=True, capture_output=True)
    return lambda *a: subprocess.run([out] + [str(int(x)) for x in a], check=True, capture_output=True,
                                     text=True).stdout.strip() == "1"


@pytest.mark.parametrize("n,steps", [(0, 5), (1, 1), (4096, 16383), (4096, 16384), (4097, 16383), (1 << 26, 1), (1 << 25, 1),
                                     (1 << 30, (1 << 31) - 1), ((1 << 30) - 1, 1 << 30), (1, (1 << 31) - 1)])
@pytest.mark.parametrize("ref", [False, True])
@pytest.mark.parametrize("limit", [0, 1, GIB, 64 * GIB, (1 << 64) - 1])
def test_the_rule_counts_every_byte(fits, n, steps, ref, limit):
    """Python's integers do not wrap: 2^30 bodies x 2^31 states are 2^65 bytes."""
    need = 16 * n * (steps + 1 + (steps if ref else 0))
    assert fits(n, steps, ref, limit) == (n > 0 and need <= limit)
