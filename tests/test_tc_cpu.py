"""The tensor-core line filter's integer arithmetic (csrc/slices.cuh, the tables
of csrc/k_tc.cu) run on the host against a long double convolution (no GPU
needed).  Errors are relative to the line's largest value; the bounds are the
result's own rounding (2^-53, 2^-24) times the few roundings on the way
(input, output, and for kernels of both signs their row sum)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
TOL = {"f64": 1e-15, "f64wide": 1e-15, "f64narrow": 2e-15, "f32": 3e-7}
LIMIT = {"f32": 2 ** 24}          # accumulators: exact below 2^22 (FP32 lines 2^24)


def test_filter_arithmetic(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "slices_check")
    csrc = os.path.join(ROOT, "scft_ver1.01_gb300", "csrc")
    obj = os.path.join(ROOT, "scft_ver1.01_gb300", "_build", "k_tc.cu.o")
    src = [os.path.join(ROOT, "tests", "native", "slices_check.cu")]
    src.append(obj if os.path.exists(obj) else os.path.join(csrc, "k_tc.cu"))
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17",
                    "--expt-relaxed-constexpr", "-I" + os.path.join(ROOT, "include"), "-I" + csrc,
                    "-o", exe] + src, check=True, capture_output=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    rows = [line.split() for line in r.stdout.splitlines()]
    assert len(rows) >= 46
    for kind, n, err, acc in rows:
        assert float(err) < TOL[kind], (kind, n, err)
        assert float(acc) < LIMIT.get(kind, 2 ** 22), (kind, n, acc)
