"""divide_by (csrc/divide.cuh), the division of the red-black updates by a kept reciprocal, compiled for the host: against
the IEEE quotient for every significand of a binade, dense steps through all magnitudes, subnormal quotients, zeros,
infinities and NaN. The CUDA build rounds every operation by itself (-fmad=false), as this one does."""

import ctypes
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "continuum_liquid_b200" / "csrc"

SOURCE = r"""
#include "divide.cuh"
#include <cstdint>
#include <cstring>
static float of(uint32_t u) { float f; std::memcpy(&f, &u, 4); return f; }
static uint32_t bits(float f) { uint32_t u; std::memcpy(&u, &f, 4); return u; }
// Mismatches over x = first, first + step, ... (bit patterns, both signs). A subnormal quotient half way between two
// neighbours may be either of them.
extern "C" long mismatches(int divisor, uint32_t first, uint32_t last, uint32_t step) {
    const volatile float d = (float)divisor;
    const float r = 1.0f / d;
    long bad = 0;
    for (uint64_t u = first; u <= last; u += step)
        for (uint32_t sign = 0; sign < 2; ++sign) {
            const float x = of((uint32_t)u | sign << 31), got = clb::divide_by(x, d, r), want = x / d;
            if (bits(got) == bits(want) || (got != got && want != want)) continue;
            // a tie: twice the quotient is odd in units of 2^-149, and got is the other neighbour
            const double units = (double)x / (double)divisor * 0x1p149;
            const bool tie = units - (double)(long long)units == (units < 0 ? -0.5 : 0.5) &&
                             (units < 0 ? -units : units) < 0x1p23 && (double)x == units * 0x1p-149 * divisor;
            const double off = (double)got * 0x1p149 - units;
            if (!tie || (off < 0 ? -off : off) != 0.5) ++bad;
        }
    return bad;
}
"""


@pytest.fixture(scope="module")
def mismatches(tmp_path_factory):
    folder = tmp_path_factory.mktemp("divide")
    source = folder / "divide.cpp"
    source.write_text(SOURCE)
    library = folder / "divide.so"
    flags = ["-O2", "-std=c++17", "-ffp-contract=off", "-fno-fast-math", "-shared", "-fPIC", f"-I{CSRC}"]
    subprocess.run(["g++", *flags, "-o", str(library), str(source)], check=True)
    f = ctypes.CDLL(str(library)).mismatches
    f.restype = ctypes.c_long
    f.argtypes = [ctypes.c_int, ctypes.c_uint32, ctypes.c_uint32, ctypes.c_uint32]
    return f


@pytest.mark.parametrize("divisor", [1, 2, 3, 4, 5, 6, 7, 9, 10, 11, 13, 22, 24, 96, 383, 1000, 1536, 12289, 24576, 32767, 32768])
def test_every_significand(mismatches, divisor):
    assert mismatches(divisor, 0x3F800000, 0x3FFFFFFF, 1) == 0


@pytest.mark.parametrize("divisor", list(range(1, 97)) + [383, 384, 1536, 6143, 24576, 32767, 32768])
def test_all_magnitudes(mismatches, divisor):
    assert mismatches(divisor, 0, 0x7FFFFFFF, 29989) == 0           # zero to infinity and NaN
    assert mismatches(divisor, 0x7F7FFF00, 0x7F800100, 1) == 0      # around infinity
    assert mismatches(divisor, 0, 40000, 1) == 0                    # the smallest
    assert mismatches(divisor, 0x00800000, 0x0C000000, 9973) == 0   # where the quotient becomes subnormal
