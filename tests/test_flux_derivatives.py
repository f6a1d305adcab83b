"""The tangent-linear model's flux derivative against the flux on dual numbers,
over every branch of the eigenvalues and of the entropy fix."""
import os
import re
import shutil
import subprocess

import pytest

from conftest import ROOT


def test_flux_derivative_matches_dual_numbers(tmp_path):
    """Both evaluations have about 60 dependent roundings of 1.1e-16, each of a
    term no larger than the sums of sizes that the difference is divided by:
    2e-14."""
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("no nvcc")
    exe = str(tmp_path / "flux_derivative_check")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-O2", "-std=c++17", "--expt-relaxed-constexpr",
                    "-I", os.path.join(ROOT, "vortex-transport_b200", "csrc"),
                    os.path.join(ROOT, "tests", "flux_derivative_check.cu"), "-o", exe],
                   check=True, capture_output=True, text=True, timeout=600)
    out = subprocess.run([exe], check=True, capture_output=True, text=True, timeout=120).stdout
    m = dict(re.findall(r"(\w+) ([\d.e+-]+)", out))
    assert int(m["used"]) > 100000, out
    for branch in ("fixed", "usual", "general"):
        assert int(m[branch]) > 5000, out
    for branch in ("between", "l0_fixed", "l1_fixed"):
        assert int(m[branch]) > 100, out
    assert float(m["worst"]) <= 2e-14, out
