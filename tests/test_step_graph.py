"""Capture of steps into a graph (tetfit_b200/csrc/step_graph.hpp) when the
runtime refuses it, through a small C++ checker with a fake runtime."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_refused_capture_leaves_nothing_behind(tmp_path):
    cxx = os.environ.get("CXX") or shutil.which("g++")
    if not cxx:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "step_graph_check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-Wall", os.path.join(HERE, "step_graph_check.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
