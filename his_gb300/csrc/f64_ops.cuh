// Float64 building blocks for GB300, whose FP64 pipe takes one warp instruction per 19
// SM cycles (64 cycles per instruction for one warp, whatever its instruction-level
// parallelism; measured with clock64 loops), against 2 for a 64-bit integer compare and
// select.  Every kernel on float64 data is bound by the number of FP64 instructions, so
// comparisons, signs, minima and maxima are taken on the bit patterns, quotients that
// share a denominator share its reciprocal, and powers are products and roots
// (pow(h, 4) costs 88 FP64 instructions, pow(h, 4/3) 87, cbrt 12, a division 7.4, a
// square root 7.5, a reciprocal 4.5).
//
// NaN: the predicates are false for NaN and the selections keep it, as the IEEE
// comparisons they stand for do.
#pragma once
#include <cuda_runtime.h>

namespace his {

constexpr unsigned long long F64_SIGN = 0x8000000000000000ull;
constexpr unsigned long long F64_INF = 0x7ff0000000000000ull;

__device__ __forceinline__ unsigned long long f64_bits(double x) { return (unsigned long long)__double_as_longlong(x); }
__device__ __forceinline__ double f64_of(unsigned long long u) { return __longlong_as_double((long long)u); }

// x > 0 and x < 0
__device__ __forceinline__ bool f64_pos(double x) { return f64_bits(x) - 1ull < F64_INF; }
__device__ __forceinline__ bool f64_neg(double x) { return (f64_bits(x) ^ F64_SIGN) - 1ull < F64_INF; }
// x >= b for a bound b > 0
__device__ __forceinline__ bool f64_ge_pos(double x, double b) {
    return f64_bits(x) - f64_bits(b) <= F64_INF - f64_bits(b);
}
// |x| < b for a bound b > 0
__device__ __forceinline__ bool f64_mag_lt(double x, double b) { return (f64_bits(x) & ~F64_SIGN) < f64_bits(b); }
// sign of x: +0 and above, -0 and below
__device__ __forceinline__ bool f64_plus(double x) { return f64_bits(x) <= F64_INF; }
__device__ __forceinline__ bool f64_minus(double x) { return (f64_bits(x) ^ F64_SIGN) <= F64_INF; }

__device__ __forceinline__ double f64_relu(double x) { return f64_pos(x) ? x : 0.0; }      // 0 for NaN
__device__ __forceinline__ double f64_clamp0(double x) { return f64_minus(x) ? 0.0 : x; }  // NaN stays

// Order-preserving integer of a finite or infinite double
__device__ __forceinline__ long long f64_key(double x) {
    const long long s = __double_as_longlong(x);
    return s ^ (long long)((unsigned long long)(s >> 63) >> 1);
}
__device__ __forceinline__ double f64_max(double a, double b) { return f64_key(a) < f64_key(b) ? b : a; }
__device__ __forceinline__ double f64_min(double a, double b) { return f64_key(b) < f64_key(a) ? b : a; }
// Running maximum of values a >= +0 (bit patterns: a negative a would stay); a NaN candidate is
// passed over, as a > comparison does
__device__ __forceinline__ double f64_max_run(double a, double b) {
    const unsigned long long u = f64_bits(b);
    return u > f64_bits(a) && u <= F64_INF ? b : a;
}

// minmod: the smaller magnitude with the common sign, 0 where the signs differ
__device__ __forceinline__ double f64_minmod(double a, double b) {
    const unsigned long long ua = f64_bits(a), ub = f64_bits(b);
    const unsigned long long m = (ua & ~F64_SIGN) < (ub & ~F64_SIGN) ? ua : ub;
    return (long long)(ua ^ ub) < 0 ? 0.0 : f64_of(m);
}

// a / b from r = 1 / b correctly rounded: the residual step of Markstein's theorem (IBM
// Journal of Research and Development 34 (1), 1990), which rounds the quotient correctly
// while neither it nor a is subnormal (then within 2 ulp); 3 FP64 instructions per numerator
// instead of 7.4.  An infinite quotient is kept; a zero loses its sign; an infinite b gives NaN.
__device__ __forceinline__ double f64_div(double a, double b, double r) {
    const double q = a * r;
    return (f64_bits(q) & ~F64_SIGN) == F64_INF ? q : fma(fma(-q, b, a), r, q);
}

// x^(4/3) for x > 0
__device__ __forceinline__ double f64_pow43(double x) { return x * cbrt(x); }

}  // namespace his
