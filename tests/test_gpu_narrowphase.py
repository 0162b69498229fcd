"""The register narrowphase gives the general one's manifolds, bit for bit, on random
pairs of every shape type (tests/cuda/small_check.cu, compiled here with nvcc)."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
REPO = os.path.dirname(HERE)
NVCC = os.path.join(os.environ.get("CUDA_HOME", "/usr/local/cuda"), "bin", "nvcc")


def test_small_narrowphase_matches_general(tmp_path):
    exe = str(tmp_path / "small_check")
    subprocess.run([NVCC, "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "--fmad=false", "-std=c++17",
                    "-I", os.path.join(REPO, "include"), "-I", os.path.join(REPO, "box2c_gb300", "csrc"),
                    os.path.join(HERE, "cuda", "small_check.cu"), "-o", exe], check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "MISMATCH" not in r.stdout and "status no error" in r.stdout
    counts = [int(x) for x in r.stdout.split("touching")[1].split()]
    assert min(counts) > 1000, r.stdout  # apart, one point and two points
