"""Launch shapes written as rules, compiled for the CPU."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.mark.skipif(not os.path.exists(NVCC), reason="nvcc not found")
def test_held_ctas_fit_the_sm(tmp_path):
    exe = str(tmp_path / "launch_shapes")
    src = os.path.join(HERE, "native", "launch_shapes.cu")
    subprocess.run([NVCC, "-std=c++17", "-O0", "--expt-relaxed-constexpr", "-gencode",
                    "arch=compute_100a,code=sm_100a", "-x", "cu", "-o", exe, src], check=True, capture_output=True,
                   timeout=600)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr
