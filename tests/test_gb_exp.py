"""The exponential of the GB/SA pairs against the extended-precision one, compiled for the host (its
arithmetic is FP64 multiply-adds, the same there): within 1.01 ulp over its range and past both
ends, and the library's values for infinities, NaN and what is out of range."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "protenix-dock_gb300", "csrc")


def test_gb_exp(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("g++ not available")
    exe = str(tmp_path / "gb_exp")
    subprocess.run([cxx, "-O2", "-std=c++17", "-ffp-contract=off", "-I", CSRC,
                    os.path.join(HERE, "native", "gb_exp_main.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe, "2000000"], capture_output=True, text=True, check=True).stdout.split("\n")
    assert float(out[0]) <= 1.01
    pairs = [line.split() for line in out[1:] if line]
    assert len(pairs) == 12
    for got, want in pairs:
        a, b = float(got), float(want)
        assert a == b or (a != a and b != b) or abs(a - b) <= 2.3e-16 * abs(b)
