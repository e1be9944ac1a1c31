"""The integer form of the refinement's long double comparison
(refine_incremental.cuh:350), on the CPU."""
import shutil
import subprocess
from pathlib import Path

import pytest

NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.mark.skipif(not Path(NVCC).exists(), reason="nvcc not available")
def test_below_fraction_equals_long_double(tmp_path):
    exe = tmp_path / "below_fraction"
    src = Path(__file__).with_name("below_fraction.cu")
    subprocess.run([NVCC, "-O1", "-std=c++17", "-gencode", "arch=compute_100a,code=sm_100a", "-o", str(exe), str(src)],
                   check=True, timeout=600)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout
