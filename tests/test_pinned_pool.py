"""The free list of a context's page-locked result blocks (pinned_pool.hpp): few sizes, bounded."""

import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_pool_has_few_sizes_and_a_limit(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = tmp_path / "pinned_pool_check"
    res = subprocess.run([cxx, "-std=c++17", "-O2", "-pthread", os.path.join(REPO, "tests", "pinned_pool_check.cpp"),
                          "-o", str(exe)], capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    res = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert res.returncode == 0, res.stdout
