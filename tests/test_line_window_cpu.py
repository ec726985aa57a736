"""The line passes' index arithmetic (itk-rs_gb300/csrc/line_window.hpp) never
leaves the smallest source that holds a request's taps, and gives every
requested output its taps: tests/cpp/line_window.cpp walks it on the host."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "itk-rs_gb300", "csrc")


def test_windows_stay_inside_the_source(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not found")
    exe = str(tmp_path / "line_window")
    subprocess.run([cxx, "-std=c++17", "-O2", "-I", CSRC, os.path.join(HERE, "cpp", "line_window.cpp"), "-o", exe],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    print(r.stdout)
    assert r.returncode == 0, r.stdout + r.stderr


def test_the_kernels_use_it():
    src = open(os.path.join(CSRC, "conv_lines.cu")).read()
    assert src.count("line_window(") == 2 and "line_steps(" in src and "line_at(" in src
