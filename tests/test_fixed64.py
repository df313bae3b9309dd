"""sf::fixed64 (csrc/kernels/softfp64.cuh), the Jacobi update's largest difference as a double, against the host FPU's
conversion of a 64-bit integer (round-to-nearest-even) scaled by a power of two."""
import ctypes
import os
import subprocess

import pytest

CODE = r"""
#include <cmath>
#include <cstdint>
#include "csrc/kernels/softfp64.cuh"
extern "C" long check(long n, uint64_t seed) {
    long bad = 0;
    for (long i = 0; i < n; i++) {
        seed = seed * 6364136223846793005ull + 1442695040888963407ull;
        const uint64_t r = seed ^ (seed >> 29);
        uint64_t q = (r << 7 | r >> 57) >> (i & 63);
        switch (i >> 6 & 7) {
            case 0: q = ~0ull >> (i & 63); break;                                       // all ones: carries
            case 1: q = (q | 1ull << 63) >> 11 << 11 | 0x400; break;                     // half-way
            case 2: q = ((q | 1ull << 63) >> 11 << 11 | 0x400) + (i % 3 == 0 ? 1 : -1); break;
            case 3: q &= ~0ull << (i & 63); break;                                       // few bits, and 0
        }
        const int E = 54 + (int)(r % 1900);
        const double want = std::ldexp((double)q, E - 1075);
        bad += sf::fixed64(q, E) != sf::bits(want);
    }
    return bad;
}
"""


@pytest.mark.parametrize("seed", [1, 20261205])
def test_against_the_fpu(tmp_path, seed):
    here = os.path.dirname(os.path.abspath(__file__))
    src, lib = tmp_path / "c.cpp", str(tmp_path / "c.so")
    src.write_text(CODE)
    subprocess.check_call(["g++", "-O2", "-ffp-contract=off", "-std=c++17", "-fPIC", "-shared", str(src), "-o", lib,
                           "-I" + os.path.join(here, "..", "dvm-snapshot-r6603-fork_gb300")])
    L = ctypes.CDLL(lib)
    L.check.restype = ctypes.c_long
    L.check.argtypes = [ctypes.c_long, ctypes.c_uint64]
    assert L.check(2_000_000, seed) == 0
