"""The procedural length scale and the level weights in float-float (csrc/ffmath.cuh)
against their double evaluations, on the host: the header compiles for the host with the
same float operations, and every value its rounding test accepts must round to the double
evaluation's float (tests/ffscale_check.cpp)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_float_float_length_scale_rounds_as_double(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if not cxx:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "ffscale_check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-o", exe,
                    os.path.join(HERE, "ffscale_check.cpp"), "-lm"], check=True)
    r = subprocess.run([exe, "1000000"], capture_output=True, text=True, timeout=600)
    print(r.stdout)
    assert r.returncode == 0, r.stdout + r.stderr
