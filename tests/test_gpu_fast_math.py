"""The device's table-driven expf, logf, log10f, exp10f and powf return the bits of the kernels
that define them (and that the host and the oracle evaluate): for every float argument, powf
at exponents and bases of the models (half the halo's index, 10^x) and others."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_float_functions_equal_their_kernels_for_every_float(tmp_path):
    exe = str(tmp_path / "fast_math_check")
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-fmad=false",
                    "--expt-relaxed-constexpr", "-o", exe, os.path.join(ROOT, "tests", "cpp", "fast_math_check.cu")], check=True)
    r = subprocess.run([exe, "10", "-1.385", "1.25", "0.5", "-3.3", "2", "7.5", "0.001"], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
