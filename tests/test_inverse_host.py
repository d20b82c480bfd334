"""The loop of the batch inverse's modular inverse (inverse.cuh) built for the host: its result for
canonical values and its end for every argument, 0 and the multiples of p among them."""

import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_almost_inverse_ends_and_matches(tmp_path):
    nvcc = next((c for c in (shutil.which("nvcc"), "/usr/local/cuda/bin/nvcc") if c and os.path.exists(c)), None)
    if nvcc is None:
        pytest.skip("nvcc not found")
    exe = tmp_path / "inverse_host"
    res = subprocess.run([nvcc, "-std=c++17", "-O2", "--expt-relaxed-constexpr",
                          os.path.join(REPO, "tests", "inverse_host.cu"), "-o", str(exe)],
                         capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    res = subprocess.run([str(exe), "3000"], capture_output=True, text=True, timeout=60)
    assert res.returncode == 0, res.stdout
