"""The grid walk and the fast triangle test, run on the CPU.

tests/cpp/tracer_check.cpp builds form_factors_b200/csrc/ffb_grid.cuh as plain
C++ and compares the faces its traversal finds with a scan over every face
(ray_caster/naive_cpu.cpp:65-97), for rays with direction components from 2^-60
down to the smallest float and for rays given by end points down to a billionth of
the scene away, and checks that no ray of scenes from the smallest to
the largest floats reads outside the cell table.  Once more under the compiler's
checks of undefined arithmetic: cell indices wrap modulo 2^32.  Tolerance: none."""
import os
import shutil
import subprocess

import pytest

from form_factors_b200 import build

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
@pytest.mark.parametrize("checks", [[], ["-fsanitize=signed-integer-overflow,bounds,shift", "-fno-sanitize-recover"]],
                         ids=["plain", "checked"])
def test_walk_equals_brute_force(tmp_path, checks):
    exe = str(tmp_path / "tracer_check")
    include = os.path.join(os.path.dirname(os.path.dirname(build.nvcc())), "include")
    subprocess.run(["g++", "-std=c++17", "-O1", "-frounding-math", "-ffp-contract=off", "-w"] + checks + ["-I", build.CSRC, "-I",
                    include, "-o", exe, os.path.join(HERE, "cpp", "tracer_check.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "mismatches 0" in r.stdout
