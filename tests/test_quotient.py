"""The quotients by fused multiply-adds (dasha_b200/csrc/quotient.h) have the division's bits: over() by 3 and 6 in both
precisions and div_by() by general divisors, over random mantissas of every exponent, the ends of the binades, all low
subnormals, both sides of the guards, dividends next to quotients and to their middles, zeros, infinities and NaN.  The
check (tests/quotient_check.cpp) runs here with the host's fma and, marked gpu, on the device."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
SRC = os.path.join(ROOT, "tests", "quotient_check.cpp")
INC = "-I" + os.path.join(ROOT, "dasha_b200", "csrc")


def _run(exe):
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "over<float> bad=0 over<double> bad=0 div_by bad=0" in r.stdout


def test_quotients_have_the_divisions_bits(tmp_path):
    exe = str(tmp_path / "quotient_check")
    subprocess.run(["g++", "-O2", "-std=c++17", "-ffp-contract=off", INC, "-o", exe, SRC], check=True)
    _run(exe)


@pytest.mark.gpu
def test_quotients_have_the_divisions_bits_on_the_device(tmp_path):
    exe = str(tmp_path / "quotient_check_gpu")
    subprocess.run(["nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-O3", "-std=c++17", "-x", "cu", INC, "-o", exe, SRC],
                   check=True)
    _run(exe)
