// FP64 logarithm, reciprocal and reciprocal square root of the pair sums, without the library
// functions' branches.  All for arguments between 2^-1007 and 2^992 (in_range64; callers take the library's
// functions elsewhere: zeros, denormals, infinities and NaN keep their results).
//
// ln x by a table and a short polynomial (P. T. P. Tang, Table-driven implementation of the
// logarithm function in IEEE floating-point arithmetic, ACM TOMS 16(4), 1990): x = 2^k m with
// m in [3/4, 3/2), c the reciprocal of the centre of m's interval (256 intervals; 1 for the
// two that meet at m = 1, so that ln x keeps its relative accuracy there), r = m c - 1 with
// |r| <= 2^-9 (2^-8 at 1): ln x = k ln 2 - ln c + ln(1 + r), the last by its series to r^7 / 7
// (the next term is below 2^-67).  12 FP64 operations and one 16-byte read.
//
// 1 / x and x^(-1/2) from the hardware's approximations y (about 2^-20) by one step of third
// order: y (1 + e + e^2) with e = 1 - x y, and y (1 + e / 2 + 3 e^2 / 8) with e = 1 - x y^2; the
// errors are of the order of e^3.
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

__device__ __forceinline__ double log64(double x, const double2* table) {
    const int h = __double2hiint(x), k = (h - 0x3fe80000) >> 20, hm = h - (k << 20);
    const double m = __hiloint2double(hm, __double2loint(x));
    const double2 t = table[(hm - 0x3fe80000) >> 12];
    // k as a double: 2^52 + 2^31 + k from its bits
    const double kd = __hiloint2double(0x43300000, k ^ (int)0x80000000) - 4503601774854144.0;
    const double r = fma(m, t.x, -1.0);
    double q = fma(r, 1.0 / 7.0, -1.0 / 6.0);
    q = fma(r, q, 1.0 / 5.0);
    q = fma(r, q, -1.0 / 4.0);
    q = fma(r, q, 1.0 / 3.0);
    q = fma(r, q, -0.5);
    // ln 2 in two parts, the first of 42 bits (its multiples by k are exact)
    const double head = fma(kd, 0x1.62e42fefa3800p-1, t.y) + r;
    return head + fma(r * r, q, kd * 0x1.ef35793c76730p-45);
}

__device__ __forceinline__ double reciprocal64(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

__device__ __forceinline__ double rsqrt64(double x) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-(x * y), y, 1.0);
    return fma(y, e * fma(e, 0.375, 0.5), y);
}

// The same for every argument.
__device__ __forceinline__ double rsqrt_any(double x) { return in_range64(x) ? rsqrt64(x) : rsqrt(x); }
__device__ __forceinline__ double reciprocal_any(double x) {
    return in_range64(x) ? reciprocal64(x) : 1.0 / x;
}
