"""Host threads of a call: no start that fails and no exception in one of them ends the process."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_failed_starts_and_exceptions(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no host compiler")
    exe = str(tmp_path / "threads_check")
    subprocess.run([cxx, "-O1", "-std=c++17", "-pthread", "-o", exe, os.path.join(HERE, "threads_check.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
