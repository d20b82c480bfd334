"""The host thread pool of the MSM combination (host_pool.hpp): a run that waits for its data holds
the pool against nobody."""

import os
import shutil
import subprocess

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_waiting_calls_hold_nobody(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = tmp_path / "host_pool_check"
    res = subprocess.run([cxx, "-std=c++17", "-O2", "-pthread", os.path.join(REPO, "tests", "host_pool_check.cpp"), "-o",
                          str(exe)], capture_output=True, text=True)
    assert res.returncode == 0, res.stderr
    res = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert res.returncode == 0, res.stdout
