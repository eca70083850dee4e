"""The square root of the FP64 direct sum against CUDA's, over the whole range of
its arguments (sums of squares from 1e-300 up)."""
import os
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")


def build(path):
    subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17",
                    "-I", os.path.join(REPO, "fastlinkingnumbers_b200", "csrc"),
                    os.path.join(REPO, "tests", "cpp", "root_check.cu"), "-o", path], check=True)
    return path


@pytest.mark.gpu
def test_root_is_within_an_ulp(tmp_path):
    out = subprocess.run([build(str(tmp_path / "root_check"))], check=True, capture_output=True, text=True, timeout=120)
    ulps, at, approx, approx_at = out.stdout.split()
    print(f"largest difference {ulps} ulp (at {at}); approximation {approx} x 2^-19 (at {approx_at})")
    assert float(approx) < 1.0
    assert int(ulps) <= 1
