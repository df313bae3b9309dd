"""The FP32-limb arithmetic of the Jacobi and heat kernels (csrc/kernels/fixlimb.cuh) is bit-identical to the host
FPU: sums of up to six non-negative doubles, rounded after every addition, and their quotients by 6 and 4."""
import ctypes
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def hostlib(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("fx") / "libfxcheck.so")
    subprocess.check_call(["g++", "-O2", "-ffp-contract=off", "-frounding-math", "-std=c++17", "-fPIC", "-shared",
                           os.path.join(HERE, "fixlimb_check.cpp"), "-o", out])
    L = ctypes.CDLL(out)
    for f in (L.fixlimb_check, L.fixlimb_check_range, L.fixlimb_check_round63):
        f.restype = ctypes.c_long
    L.fixlimb_check.argtypes = L.fixlimb_check_round63.argtypes = [ctypes.c_long, ctypes.c_uint64]
    return L


@pytest.mark.parametrize("seed", [1, 20261206])
def test_sums_and_quotients_match_the_host_fpu(hostlib, seed):
    assert hostlib.fixlimb_check(1_000_000, seed) == 0


def test_splitting_refuses_what_the_limbs_cannot_hold(hostlib):
    assert hostlib.fixlimb_check_range() == 0


@pytest.mark.parametrize("seed", [2, 20261207])
def test_rounding_of_integers_matches_the_host_fpu(hostlib, seed):
    """The heat kernel's S - 4 src: a signed 63-bit integer rounded once to a double."""
    assert hostlib.fixlimb_check_round63(4_000_000, seed) == 0
