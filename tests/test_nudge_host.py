"""The nudge rule of the coarse results, compiled for the host (nvcc, no GPU)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "ampcor_b200", "csrc")
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")


@pytest.mark.skipif(not (os.path.exists(NVCC) or shutil.which("nvcc")), reason="nvcc not found")
def test_nudged_corners_stay_inside(tmp_path):
    exe = str(tmp_path / "nudge_host_check")
    subprocess.run([NVCC, "-std=c++17", "-O2", "-arch=sm_100a", "-I", CSRC, "-o", exe,
                    os.path.join(HERE, "nudge_host_check.cu")], check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
