"""The products of field.cuh on factors that nothing has reduced, built for the host
(tests/field_any_host.cu), against 128-bit host arithmetic."""

import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_products_of_unreduced_factors(tmp_path):
    nvcc = next((c for c in (shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc") if c and os.path.exists(c)), None)
    if nvcc is None:
        pytest.skip("nvcc not found")
    exe = tmp_path / "field_any_host"
    res = subprocess.run([nvcc, "-std=c++17", "-O2", "--expt-relaxed-constexpr",
                          os.path.join(REPO, "tests", "field_any_host.cu"), "-o", str(exe)],
                         capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    res = subprocess.run([str(exe), "300000"], capture_output=True, text=True)
    assert res.returncode == 0, res.stdout
