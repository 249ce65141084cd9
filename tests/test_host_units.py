"""Host-side pieces of the library that need neither CUDA nor a GPU, compiled
with the host compiler and run against fakes (tests/cpp/*_test.cpp)."""
import os
import subprocess

import pytest

CPP = os.path.join(os.path.dirname(os.path.abspath(__file__)), "cpp")


@pytest.mark.parametrize("name", ["host_slots", "tune_pick", "l96_forms"])
def test_host_unit(name, tmp_path):
    exe = str(tmp_path / name)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-Wall", "-Werror", os.path.join(CPP, name + "_test.cpp"),
                    "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout == "ok\n", r.stdout + r.stderr
