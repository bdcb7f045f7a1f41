"""The float64 kernels' quotient from a shared reciprocal (f64_ops.cuh) against a / b, compiled
for the host from the library's own header (its device intrinsics as their host equals)."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parents[1] / "his_gb300" / "csrc"

STUB = """#pragma once
#include <cmath>
#include <cstring>
using std::fma; using std::cbrt;
#define __device__
#define __forceinline__ inline
static inline long long __double_as_longlong(double x) { long long u; std::memcpy(&u, &x, 8); return u; }
static inline double __longlong_as_double(long long u) { double x; std::memcpy(&x, &u, 8); return x; }
"""

# 1 / b is correctly rounded by the host's division, as the device's reciprocal is.  Operands and
# quotients away from the ends of the range must agree in every bit; where the quotient or the
# numerator is subnormal the residual is rounded, by at most an ulp of the quotient each for it
# and for the product it corrects.
MAIN = r"""#include <cstdio>
#include <cstdint>
#include <initializer_list>
#include <limits>
#include "f64_ops.cuh"
using namespace his;
static uint64_t s = 88172645463325252ull;
static uint64_t rnd() { s ^= s << 13; s ^= s >> 7; s ^= s << 17; return s; }
static double num(int lo, int hi) {
    uint64_t m = rnd() & ((1ull << 52) - 1);
    switch (rnd() & 7) { case 0: m = 0; break; case 1: m = (1ull << 52) - 1; break; case 2: m &= 7; break; }
    return std::ldexp(1.0 + std::ldexp((double)m, -52), lo + (int)(rnd() % (uint64_t)(hi - lo + 1))) * ((rnd() & 1) ? 1 : -1);
}
static double div(double a, double b) { return f64_div(a, b, 1.0 / b); }
int main() {
    const double inf = std::numeric_limits<double>::infinity(), nan = std::numeric_limits<double>::quiet_NaN();
    long bad = 0, sub = 0, special = 0;
    for (int k = 0; k < 4000000; ++k) {
        const double a = num(-300, 300), b = num(-300, 300);
        bad += div(a, b) != a / b;
    }
    for (int k = 0; k < 2000000; ++k) {                  // subnormal numerators and quotients
        const double b = num(-30, 30), a = (k & 1) ? std::ldexp((double)(rnd() & 0xfffffffffffffull), -1074) : num(-1070, -990);
        const double q = a / b, ulp = std::nextafter(std::fabs(q), inf) - std::fabs(q);
        sub += !(std::fabs(div(a, b) - q) <= 2.0 * ulp);
    }
    for (double b : {1e-3, 1.0, 7.0, -3.5, 1e300}) {
        special += div(0.0, b) != 0.0 || div(-0.0, b) != 0.0;
        special += div(inf, b) != inf / b || div(-inf, b) != -inf / b;
        special += div(nan, b) == div(nan, b);
        special += div(b, 0.0) != b / 0.0 || div(b, -0.0) != b / -0.0;
        special += div(b, nan) == div(b, nan);
        special += div(b, inf) == div(b, inf);           // (NaN: the states divided by have ended by then)
    }
    special += div(0.0, 0.0) == div(0.0, 0.0) || div(inf, 0.0) != inf;
    std::printf("%ld %ld %ld\n", bad, sub, special);
}
"""


def test_f64_div_is_the_correctly_rounded_quotient(tmp_path):
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    (tmp_path / "cuda_runtime.h").write_text(STUB)
    (tmp_path / "main.cpp").write_text(MAIN)
    subprocess.run(["g++", "-std=c++17", "-O2", "-ffp-contract=off", f"-I{tmp_path}", f"-I{CSRC}", "-x", "c++",
                    str(tmp_path / "main.cpp"), "-o", str(tmp_path / "main")], check=True)
    out = subprocess.run([str(tmp_path / "main")], check=True, capture_output=True, text=True).stdout
    assert out.split() == ["0", "0", "0"], out
