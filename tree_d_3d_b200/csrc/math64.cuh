// FP64 logarithm and reciprocal of the direct log sums, from one table look-up and without the
// library functions' branches, for arguments of [2^-1007, 2^993) (in_range64; callers take the
// library's functions and division elsewhere: zeros, denormals, infinities and NaN keep their
// results).
//
// ln x by a table and a short polynomial (P. T. P. Tang, Table-driven implementation of the
// logarithm function in IEEE floating-point arithmetic, ACM TOMS 16(4), 1990): x = 2^k m with
// m in [3/4, 3/2), c the reciprocal of the centre of m's interval (256 intervals; 1 for the
// two that meet at m = 1, so that ln x keeps its relative accuracy there), r = m c - 1 with
// |r| <= 2^-9 (2^-8 at 1): ln x = k ln 2 - ln c + ln(1 + r), the last by its series to r^7 / 7
// (the next term is below 2^-67).  12 FP64 operations and one 16-byte read.
//
// 1 / x from the same c and r, by the geometric series: m c = 1 + r, so
//   1 / x = 2^-k c / (1 + r),  1 / (1 + r) = 1 - r g,  g = (1 - r)(1 + r^2)(1 + r^4) / (1 - r^8).
// Without its last factor (within 2^-64 of 1) and with its four roundings g is within 2^-50.6;
// 2^-k c is exact, so C - C r g in one multiply-add has an error of 1/2 ulp and of |r| times g's
// and the product's and of the rounding of r (2^-61): under 0.52 ulp (0.508 at the most over
// 20 million arguments, half of them beside a power of two, on the CPU).
#pragma once

#include "common.cuh"

constexpr int LOG64_SIZE = 256;

__device__ __forceinline__ bool in_range64(double x) {
    return (unsigned)(__double2hiint(x) - 0x01000000) < 0x7d000000u;
}

// The table (c, -ln c), filled by the block's threads; the caller synchronises.
__device__ __forceinline__ void fill_log64(double2* table) {
    for (int t = threadIdx.x; t < LOG64_SIZE; t += blockDim.x) {
        const double a = __hiloint2double(0x3fe80000 + (t << 12), 0);
        const double b = __hiloint2double(0x3fe80000 + ((t + 1) << 12), 0);
        const double c = a == 1.0 || b == 1.0 ? 1.0 : 1.0 / (0.5 * (a + b));
        table[t] = make_double2(c, -log(c));
    }
}

// 1 / x and, with LN, ln x.
template <bool LN>
__device__ __forceinline__ void log_reciprocal64(double x, const double2* table, double& ln,
                                                 double& inv) {
    const int h = __double2hiint(x), k = (h - 0x3fe80000) >> 20, hm = h - (k << 20);
    const double m = __hiloint2double(hm, __double2loint(x));
    const double2 t = table[(hm - 0x3fe80000) >> 12];
    const double r = fma(m, t.x, -1.0), s = r * r;
    if (LN) {
        // k as a double: 2^52 + 2^31 + k from its bits
        const double kd = __hiloint2double(0x43300000, k ^ (int)0x80000000) - 4503601774854144.0;
        double q = fma(r, 1.0 / 7.0, -1.0 / 6.0);
        q = fma(r, q, 1.0 / 5.0);
        q = fma(r, q, -1.0 / 4.0);
        q = fma(r, q, 1.0 / 3.0);
        q = fma(r, q, -0.5);
        // ln 2 in two parts, the first of 42 bits (its multiples by k are exact)
        const double head = fma(kd, 0x1.62e42fefa3800p-1, t.y) + r;
        ln = head + fma(s, q, kd * 0x1.ef35793c76730p-45);
    }
    const double c = __hiloint2double(__double2hiint(t.x) - (k << 20), __double2loint(t.x));
    const double a = 1.0 + s, b = fma(s * s, a, a);  // (1 + r^2)(1 + r^4)
    const double g = fma(-r, b, b);
    inv = fma(c, -r * g, c);
}
