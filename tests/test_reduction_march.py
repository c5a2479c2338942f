"""The diagnostics' reduction marches along z and asks L2 for planes ahead of their
loads: none of them lies outside the grid (checked on the host, no GPU involved)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def test_prefetched_planes_lie_in_the_grid(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "reduction_march_check")
    subprocess.run([nvcc, "-std=c++17", "-O1", "-I", os.path.join(ROOT, "wavedm.jl_gb300", "csrc"),
                    os.path.join(HERE, "reduction_march_check.cu"), "-o", exe], check=True, capture_output=True, timeout=600)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip().splitlines()[-1] == "ALL OK", r.stdout
