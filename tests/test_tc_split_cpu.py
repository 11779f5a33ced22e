"""The rule by which the 64-bit tensor-core kernels of 16 points per thread are used
or left out (csrc/tc_core.cuh, split_fits), against its meaning: the block's
registers are those it was launched with, the issuing warpgroup only gives some
back, the computing ones only take.  A compiler's other register count must leave
the kernels out, not fail the creation of every context."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_register_split(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "split_check")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17",
                    "--expt-relaxed-constexpr", "-I" + os.path.join(ROOT, "include"),
                    "-I" + os.path.join(ROOT, "scft_ver1.01_gb300", "csrc"), "-o", exe,
                    os.path.join(ROOT, "tests", "native", "split_check.cu")],
                   check=True, capture_output=True)
    out = subprocess.run([exe], capture_output=True, text=True, check=True).stdout.splitlines()
    take, give = map(int, out[0].split())
    assert take % 8 == 0 and give % 8 == 0
    seen = set()
    for line in out[1:]:
        regs, c, fits = map(int, line.split())
        want = give <= regs <= take and c * (take - regs) <= regs - give
        assert bool(fits) == want, (regs, c)
        seen.add((regs, c, fits))
    assert all((96, c, 1) in seen for c in (2, 3, 4)) and (94, 4, 0) in seen
