"""The force windows' runs of cells (hal-cpp_gb300/csrc/agent_window.h), built
for the CPU under AddressSanitizer and UndefinedBehaviorSanitizer: the cells and
their order are the CPU backend's for agents anywhere, far outside the grid
included, and no run reaches past the cell offsets."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_window_runs(tmp_path):
    cxx = shutil.which("g++")
    if cxx is None:
        pytest.skip("g++ not found")
    exe = str(tmp_path / "window_driver")
    build = subprocess.run([cxx, "-std=c++17", "-O1", "-g", "-fsanitize=address,undefined", "-fno-sanitize-recover=all",
                            "-I", os.path.join(ROOT, "hal-cpp_gb300", "csrc"),
                            os.path.join(ROOT, "tests", "sanitize", "window_driver.cpp"), "-o", exe],
                           capture_output=True, text=True)
    if build.returncode != 0 and "asan" in (build.stderr + build.stdout).lower():
        pytest.skip("sanitizer runtime not available: " + build.stderr[-200:])
    assert build.returncode == 0, build.stderr
    run = subprocess.run([exe], capture_output=True, text=True, timeout=600)
    assert run.returncode == 0, run.stdout + run.stderr
    assert run.stdout.startswith("ok "), run.stdout
