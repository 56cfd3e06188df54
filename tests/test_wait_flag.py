"""The wait for published results (flock_gb300/csrc/gpu/wait.h), compiled with the host compiler and run
as a child process."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_rounds_are_bounded_and_stages_last_as_long_as_the_stream(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = tmp_path / "wait_flag"
    subprocess.run([cxx, "-O2", "-std=c++17", "-pthread", "-o", str(exe), os.path.join(HERE, "native", "wait_flag.cc")],
                   check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout + out.stderr
    assert "failures 0" in out.stdout
