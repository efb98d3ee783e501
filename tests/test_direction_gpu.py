"""The conjugate-gradient direction step inside the operator (sipg_op::apply_direction), through a
C++ program against the library: its result, and the refusal of misaligned vectors."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LIBDIR = os.path.join(ROOT, "ins-solver_b200")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


def _build(tmp_path):
    exe = str(tmp_path / "direction_check")
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-Wall", "-Werror", "-I", os.path.join(CUDA, "include"),
                        os.path.join(ROOT, "tests", "cpp", "direction_check.cpp"), "-o", exe, "-L", LIBDIR, "-lsipg_b200",
                        "-Wl,-rpath," + LIBDIR, "-L", os.path.join(CUDA, "lib64"), "-lcudart"],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return exe


def test_direction_check_compiles_and_links(tmp_path):
    _build(tmp_path)


@pytest.mark.gpu
def test_direction_step_and_its_refusals(tmp_path):
    r = subprocess.run([_build(tmp_path)], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and r.stdout.strip().endswith("OK"), r.stdout + r.stderr
