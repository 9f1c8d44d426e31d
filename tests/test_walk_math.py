"""The walk's shared arithmetic (math_b200/csrc/walk_math.hpp) against the routines it stands in for, on
the host: the finest-cell index of a point against the descent, the exit by approximate quotients
against the exact slabs, for points on, beside and between box boundaries, and the division of path and
pixel numbers by multiplication against the integer division.  Where the fast rule says it
can decide, the result must be the exact one's."""

import os
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]


def test_cell_index_and_exit_match_the_exact_routines(tmp_path):
    exe = tmp_path / "walk_math_check"
    cuda = os.environ.get("CUDA_HOME", "/usr/local/cuda")
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", "-I", str(ROOT / "math_b200" / "csrc"),
                    "-I", f"{cuda}/include", str(ROOT / "tests" / "cpp" / "walk_math_check.cpp"), "-o", str(exe)],
                   check=True, capture_output=True, text=True)
    run = subprocess.run([str(exe), "5000"], capture_output=True, text=True)
    assert run.returncode == 0, run.stdout + run.stderr
    assert run.stdout.count("located") == 4
