"""The softmax gradient's quotient (pbrt-v2_gb300/csrc/pbg_quotient.h) against
the IEEE division over the range that it claims; host build of the header that
the training kernel includes (fused multiply-adds and divisions are IEEE's on
both)."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


def test_quotient_is_the_division(tmp_path):
    cxx = shutil.which("g++") or shutil.which("c++")
    if cxx is None:
        pytest.skip("no C++ compiler")
    exe = str(tmp_path / "quotient_check")
    subprocess.check_call([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-o", exe,
                           os.path.join(HERE, "native", "quotient_check.cpp")])
    out = subprocess.run([exe, "20000000"], capture_output=True, text=True)
    assert out.returncode == 0, out.stdout
    n, unequal, outside = map(int, out.stdout.split())
    assert n == 20000000 and unequal == 0 and outside == 0
