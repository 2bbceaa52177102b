"""Step count of the refinement's last re-orthogonalisation (csrc/orth_steps.h,
used by csrc/eig_refine.cu), compiled by the host compiler.

One step squares the deviation from orthogonality, 16·em⁴ after the step that is
always taken; from em = ½ on the squares never get below any bound.  The child
process has a time limit: a count that does not end is the failure looked for.
"""
import math
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "tensornetworkad.jl_gb300" / "csrc"


@pytest.fixture(scope="module")
def steps(tmp_path_factory):
    cxx = shutil.which("g++") or pytest.skip("no host C++ compiler")
    d = tmp_path_factory.mktemp("orth")
    (d / "m.cpp").write_text('#include <cstdio>\n#include <cstdlib>\n#include "orth_steps.h"\n'
                             "int main(int, char** a) { std::printf(\"%d\", tnad::orth_steps(std::strtof(a[1], nullptr))); }\n")
    subprocess.run([cxx, "-std=c++17", "-Wall", "-Werror", f"-I{CSRC}", "-o", str(d / "m"), str(d / "m.cpp")], check=True)
    return lambda em: int(subprocess.run([str(d / "m"), repr(em)], capture_output=True, text=True, timeout=20, check=True).stdout)


@pytest.mark.parametrize("em", [0.11, 0.49, 0.5, 0.51, 1.0, 3.0, 1e30, math.inf, math.nan])
def test_no_correction_is_refused(steps, em):
    assert steps(em) == 0


@pytest.mark.parametrize("em", [0.0, 2e-8, 1e-5, 1e-4, 1e-3, 1e-2, 0.05, 0.1])
def test_steps_reach_rounding(steps, em):
    k = steps(em)
    assert 1 <= k <= 4
    assert (16 * em**4) ** (2 ** (k - 1)) <= 1e-16


def test_the_refinement_uses_it():
    src = (CSRC / "eig_refine.cu").read_text()
    assert "orth_steps(em)" in src and "d *= d" not in src
