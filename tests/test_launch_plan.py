"""The launch shapes and buffer sizes of flock_gb300/csrc/gpu/plan.h at any SM count: compiled with
the host compiler and run as a child process."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_launches_fit_their_buffers_at_any_sm_count(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = tmp_path / "launch_plan"
    subprocess.run([cxx, "-O2", "-std=c++17", "-o", str(exe), os.path.join(HERE, "native", "launch_plan.cc")], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout + out.stderr
    assert "failures 0" in out.stdout
