"""The unpacked integer adder and the integer division by an out-degree
(csrc/prx_softadd.h, compiled here for the host) against the CPU's IEEE 754
operations (tests/cpp/test_softacc.cpp)."""
import os
import shutil
import subprocess

import pytest

from conftest import PKG, ROOT


def test_unpacked_adder_and_quotient_match_ieee(tmp_path):
    if not shutil.which("g++"):
        pytest.skip("g++ not available")
    exe = str(tmp_path / "test_softacc")
    subprocess.run(["g++", "-std=c++17", "-O2", "-I", os.path.join(PKG, "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "test_softacc.cpp"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=600)
    print(r.stdout)
    assert r.returncode == 0, r.stdout + r.stderr
