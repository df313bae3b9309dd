"""The SOR step's sum of six neighbours on FP32 limbs (fx::sumDouble in csrc/kernels/fixlimb.cuh) is bit-identical to the
host FPU's, over the nine binades of its range, ties, carries into the next binade and zeros among the terms."""
import ctypes
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.parametrize("seed", [3, 20261208])
def test_sums_of_six_match_the_host_fpu(tmp_path, seed):
    out = str(tmp_path / "libsum.so")
    subprocess.check_call(["g++", "-O2", "-ffp-contract=off", "-frounding-math", "-std=c++17", "-fPIC", "-shared",
                           os.path.join(HERE, "sumlimb_check.cpp"), "-o", out])
    L = ctypes.CDLL(out)
    L.sumlimb_check.restype = ctypes.c_long
    L.sumlimb_check.argtypes = [ctypes.c_long, ctypes.c_uint64]
    assert L.sumlimb_check(1_000_000, seed) == 0
