"""Division by a known divisor (csrc/slice_common.cuh, divide_by), restated in C
as in test_constant_division.py and compared with IEEE division for EVERY
significand of the numerator, for the divisors 1 - 1/n and n/2 - 1/2 of every
box up to 192 and of the rfft axes of these boxes, and of larger ones.  A
mis-rounded quotient could be a single significand's, so none is left out."""

import ctypes
import os
import subprocess

import numpy as np
import pytest

CODE = r"""
#include <stdint.h>
#include <string.h>
#include <math.h>
long mismatches(float b, float r) {
    long bad = 0;
    for (uint32_t i = 0; i < (1u << 23); i++) {
        uint32_t u = 0x3f800000u | i;
        float a, q;
        memcpy(&a, &u, 4);
        q = a * r;
        q = fmaf(fmaf(-q, b, a), r, q);
        q = fmaf(fmaf(-q, b, a), r, q);
        bad += q != a / b;
    }
    return bad;
}
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("div")
    (d / "div.c").write_text(CODE)
    flags = "-O3 -march=native -shared -fPIC -ffp-contract=off -fno-math-errno -fno-trapping-math".split()
    subprocess.run(["gcc", *flags, "-o", str(d / "div.so"), str(d / "div.c"), "-lm"], check=True)
    L = ctypes.CDLL(str(d / "div.so"))
    L.mismatches.restype = ctypes.c_long
    L.mismatches.argtypes = [ctypes.c_float, ctypes.c_float]
    return L


def _divisors():
    one, half = np.float32(1.0), np.float32(0.5)
    for n in [*range(2, 193), *range(192, 1025, 64), 201, 255, 257, 319, 321, 511, 513, 1023]:
        yield one - one / np.float32(n)
        for axis in (n, n // 2 + 1):
            if axis > 1:
                yield half * np.float32(axis) - half


def test_every_numerator(lib):
    if "fma" not in open("/proc/cpuinfo").read() and os.uname().machine == "x86_64":
        pytest.skip("no fused multiply-add on this CPU: the exhaustive run would take minutes")
    for b in sorted({float(b) for b in _divisors()}):
        assert lib.mismatches(b, float(np.float32(1.0) / np.float32(b))) == 0, b
