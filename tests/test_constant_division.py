"""Division by a known divisor through its reciprocal and two FMA corrections
(csrc/slice_common.cuh, divide_by), restated in C and compared with IEEE
division (CPU): every significand of the numerator, for the divisors
1 - 1/n and n/2 - 1/2 of small, large, odd, prime and power-of-two boxes.
Scaling a numerator by a power of two scales the whole computation, so one
binade covers them all."""

import ctypes
import subprocess

import numpy as np
import pytest

CODE = r"""
#include <stdint.h>
#include <string.h>
#include <math.h>
float divide_by(float a, float b, float r) {
    float q = a * r;
    q = fmaf(fmaf(-q, b, a), r, q);
    return fmaf(fmaf(-q, b, a), r, q);
}
long mismatches(float b, float r, uint32_t step) {
    long bad = 0;
    for (uint32_t i = 0; i < (1u << 23); i += step) {
        uint32_t u = 0x3f800000u | i;
        float a;
        memcpy(&a, &u, 4);
        bad += divide_by(a, b, r) != a / b;
    }
    return bad;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("div")
    (d / "div.c").write_text(CODE)
    subprocess.run(["gcc", "-O2", "-shared", "-fPIC", "-ffp-contract=off", "-o", str(d / "div.so"), str(d / "div.c"),
                    "-lm"], check=True)
    L = ctypes.CDLL(str(d / "div.so"))
    L.mismatches.restype = ctypes.c_long
    L.mismatches.argtypes = [ctypes.c_float, ctypes.c_float, ctypes.c_uint32]
    return L


@pytest.mark.parametrize("n", [2, 3, 5, 24, 64, 67, 96, 127, 160, 200, 251, 256, 320, 487, 512, 1000, 1024])
def test_divide_by_is_correctly_rounded(lib, n):
    one = np.float32(1.0)
    for b in (one - one / np.float32(n), np.float32(0.5) * np.float32(n) - np.float32(0.5)):
        assert lib.mismatches(float(b), float(one / b), 7) == 0
