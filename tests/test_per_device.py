"""Kernel attributes are set once per device, not once per process
(csrc/per_device.h): a context on a second device needs them as well."""
import ctypes as C
import re
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "tensornetworkad.jl_gb300" / "csrc"


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    cxx = shutil.which("g++") or pytest.skip("no host C++ compiler")
    d = tmp_path_factory.mktemp("pd")
    (d / "m.cpp").write_text('#include "per_device.h"\nstatic tnad::PerDevice p;\n'
                             'extern "C" int has(int d) { return p.has(d); }\nextern "C" void mark(int d) { p.mark(d); }\n')
    subprocess.run([cxx, "-std=c++17", "-Wall", "-Werror", "-shared", "-fPIC", f"-I{CSRC}", "-o", str(d / "m.so"),
                    str(d / "m.cpp")], check=True)
    return C.CDLL(str(d / "m.so"))


def test_each_device_is_its_own(lib):
    for dev in (0, 1, 7, 63):
        assert not lib.has(dev)
        lib.mark(dev)
        assert lib.has(dev)
    assert not lib.has(2)
    for dev in (64, 1000, -1):  # never marked
        lib.mark(dev)
        assert not lib.has(dev)


@pytest.mark.parametrize("path", sorted(CSRC.glob("*.cu")), ids=lambda p: p.name)
def test_no_process_wide_flag_guards_an_attribute(path):
    """Every cudaFuncSetAttribute stands in a block that a PerDevice guards, or is unconditional."""
    text = path.read_text()
    assert not re.search(r"static\s+(std::atomic<bool>|bool|std::once_flag)\s+\w+[^;]*;(?:(?!\n}).)*?cudaFuncSetAttribute",
                         text, re.S)
