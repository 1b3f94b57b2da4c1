"""The membrane's division by shared divisors (csrc/div.h), compiled for the
host, against the division: the bits have to be the same over the range that the
header states, for 3 and 6, for doubled masses with few and with all mantissa
bits, and for values whose quotient lies next to a rounding boundary."""
import ctypes as C
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

HARNESS = r"""
#include <cstdint>
#include <cstring>
#include <random>
#include "div.h"
using namespace irbc;
extern "C" int64_t differ(double y, int e0, int e1, int64_t n, unsigned seed) {
  std::mt19937_64 g(seed);
  const Divisor d{y, 1.0 / y};
  int64_t bad = 0;
  for (int64_t k = 0; k < n; ++k) {
    const double m = 1.0 + (double)(g() >> 12) * 0x1p-52;
    const int e = e0 + (int)(g() % (uint64_t)(e1 - e0 + 1));
    double x = std::ldexp((g() & 1) ? -m : m, e);
    if (k & 1) {
      // next to a boundary: y times the middle of two neighbouring quotients
      const double q = x / y, s = std::fabs(q), up = std::nextafter(s, HUGE_VAL);
      x = std::copysign((double)(((long double)s + ((long double)up - s) / 2) * (long double)std::fabs(y)), x);
      const int off = (int)(g() % 5) - 2;
      for (int u = 0; u < std::abs(off); ++u) x = std::nextafter(x, off < 0 ? 0.0 : (x < 0 ? -HUGE_VAL : HUGE_VAL));
    }
    const double want = x / y, got = div_by(x, d);
    bad += std::memcmp(&want, &got, sizeof(double)) != 0;
  }
  return bad;
}
extern "C" double one(double x, double y) { return div_by(x, Divisor{y, 1.0 / y}); }
"""


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = tmp_path_factory.mktemp("div")
    src, so = str(d / "h.cpp"), str(d / "h.so")
    with open(src, "w") as f:
        f.write(HARNESS)
    subprocess.run([os.environ.get("IRBC_CXX", "g++"), "-O2", "-std=c++17", "-ffp-contract=off", "-shared", "-fPIC",
                    "-I" + os.path.join(ROOT, "irbc-code_b200", "csrc"), src, "-o", so], check=True)
    L = C.CDLL(so)
    L.differ.restype = C.c_int64
    L.differ.argtypes = [C.c_double, C.c_int, C.c_int, C.c_int64, C.c_uint]
    L.one.restype = C.c_double
    L.one.argtypes = [C.c_double, C.c_double]
    return L


# 2 m of the default mass; full mantissas, all ones among them; next to powers of two
DIVISORS = [3.0, 6.0, 20.0, 2.0 / 3.0, 0.2, 20.000000000000004, float.fromhex("0x1.fffffffffffffp+3"),
            float.fromhex("0x1.0000000000001p+0"), 7.123456789012345e-3, 9.87654321098765e5]


@pytest.mark.parametrize("y", DIVISORS)
def test_the_bits_of_the_division(lib, y):
    assert lib.differ(y, -20, 20, 400000, 1) == 0
    # the ends of the stated range (the quotients stay finite: |y| > 2^-8)
    assert lib.differ(y, -968, 1010, 400000, 2) == 0


def test_below_the_range_only_the_last_bit(lib):
    # (normal quotients, with a divisor of many bits)
    assert lib.differ(2.0 / 3.0, -1018, -1012, 400000, 3) > 0
    for x in (5e-310, -3.3e-305, 1e-300):
        assert lib.one(x, 7.1) == pytest.approx(x / 7.1, rel=4e-16, abs=1e-323)
