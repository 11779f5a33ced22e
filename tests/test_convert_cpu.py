"""The integer conversions between FP64, FP32 and pairs (csrc/convert.cuh) are the
casts, bit for bit: zeros, denormals, infinities, NaN, the edges of the range that
the integer steps cover, rounding ties and carries (no GPU needed)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_conversions(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "convert_check")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-O2",
                    "--expt-relaxed-constexpr", "-I" + os.path.join(ROOT, "scft_ver1.01_gb300", "csrc"),
                    "-o", exe, os.path.join(ROOT, "tests", "native", "convert_check.cu")],
                   check=True, capture_output=True)
    n, bad = map(int, subprocess.run([exe], capture_output=True, text=True, check=True).stdout.split())
    assert n > 30_000_000 and bad == 0
