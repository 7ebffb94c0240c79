"""Launch rules of the resident CG kernels (tetfit_b200/csrc/resident_choice.hpp)
through a small C++ checker built with the host compiler: what the device's
answers allow is chosen, what they refuse is left to the general kernels."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_choices_follow_the_device(tmp_path):
    cxx = os.environ.get("CXX") or shutil.which("g++")
    if not cxx:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "resident_choice_check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-Wall", os.path.join(HERE, "resident_choice_check.cpp"), "-o", exe],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
