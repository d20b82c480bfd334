"""The host's multiple of a point (host_field.hpp, proof assembly) against double-and-add: the same
point, for no more products whatever the scalar."""

import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_multiples_cost_no_more_than_double_and_add(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = tmp_path / "host_mul_check"
    res = subprocess.run([cxx, "-std=c++17", "-O2", os.path.join(REPO, "tests", "host_mul_check.cpp"), "-o", str(exe)],
                         capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    res = subprocess.run([str(exe)], capture_output=True, text=True)
    assert res.returncode == 0, res.stdout
