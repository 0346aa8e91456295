"""The boundary face reverse against dual numbers, compiled for the CPU."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.mark.skipif(not os.path.exists(NVCC), reason="nvcc not found")
def test_boundary_reverse_matches_dual_numbers(tmp_path):
    exe = str(tmp_path / "boundary_adjoint")
    src = os.path.join(HERE, "native", "boundary_adjoint.cu")
    subprocess.run([NVCC, "-std=c++17", "-O1", "-gencode", "arch=compute_100a,code=sm_100a", "-x", "cu", "-o", exe,
                    src], check=True, capture_output=True, timeout=300)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
