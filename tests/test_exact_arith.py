"""The integer square root, reciprocal and quotient of csrc/p3t_exact.cuh are
the IEEE ones, bit for bit (no tolerance): against g++'s operations on the CPU,
and on the device against the host's."""
import os
import subprocess

import pytest

from gplum_gb300 import build

SRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "cxx", "exact_arith.cpp")


def _run(cmd, exe, n):
    r = subprocess.run(cmd + ["-I", build.CSRC, "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([exe, str(n)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr


def test_integer_forms_round_as_ieee(tmp_path):
    _run(["g++", "-O2", "-std=c++17", SRC], str(tmp_path / "exact"), 3000000)


@pytest.mark.gpu
def test_integer_forms_round_as_ieee_on_the_device(gpu, tmp_path):
    _run([build._nvcc(), *build.ARCH, "-O2", "-std=c++17", "-fmad=false", "-x", "cu", SRC], str(tmp_path / "exact"), 100000)
