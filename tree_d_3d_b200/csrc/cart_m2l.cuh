// M2L of the softened Coulomb kernel with Cartesian expansions of orders up to 16, a lane
// per translation (K/cart_m2l_host/cart_m2l_host_pyccel.py:16-80; higher orders:
// fmm_cart.cu).
//
// Scaled form: with m~_a = (-1)^|a| m_a / (a_x! a_y!) and A~_g = D^g f(t) the derivatives of
// f = (|r|^2 + eps^2)^(-1/2), T_b = T~_b / (b_x! b_y!), T~_b = sum_a m~_a A~_(a+b) over
// |a| + |b| <= p.
//
// What bounds it: the C(p + 4, 4) products of a translation (1820 at p = 12) on the FP64
// (FP32) pipe.  A lane therefore takes one translation whole and keeps what a product needs
// in registers: the sums T~_b, and two neighbouring degrees of A = A~ / (g_x! g_y!), which
// the recurrence
//   A_g = -(1 / (n R^2)) ((2n - 1) (t_x A_(g-ex) + t_y A_(g-ey)) + (n - 1) (A_(g-2ex) + A_(g-2ey)))
// advances in place, so A never goes to memory.  The moments come from shared memory, 4 to 6
// products per value read (with A and the moments both there the reads cost twice the
// products' time).
//
// Measured (1M clustered particles, theta 0.5, 12.6M translations, records included; a lane per
// coefficient run with both operands in shared memory before): p = 12 FP64 18.6 -> 5.6 ms, FP32
// 13.2 -> 4.5 ms (100k particles, the two of a backward step: 2.3 -> 0.9 ms).
//
// Work: a warp walks its rows with four lanes per row (walk_rows); a lane keeps its sums
// across the row, at whose end the group's 4 lanes are added through shared memory and each
// lane adds a quarter of the coefficients to the locals: the same bits every run.
//
// Mixed precision (T = float): moments in a unit of length near the source cell's half-width,
// sums in one near the destination's, both powers of two; see unit_of() and translate().
#pragma once

#include "row_groups.cuh"

#include <type_traits>
#include <utility>

namespace {

__host__ __device__ constexpr int tri(int n) { return n * (n + 1) / 2; }
__host__ __device__ constexpr double factorial(int n) { return n < 2 ? 1.0 : n * factorial(n - 1); }
__host__ __device__ constexpr int degree_of(int i) {
    int n = 0;
    while (tri(n + 1) <= i) ++n;
    return n;
}

// f(std::integral_constant<int, 0>) ... f(std::integral_constant<int, N - 1>)
template <class F, int... I>
__device__ __forceinline__ void static_for_impl(F&& f, std::integer_sequence<int, I...>) {
    (f(std::integral_constant<int, I>{}), ...);
}
template <int N, class F>
__device__ __forceinline__ void static_for(F&& f) {
    static_for_impl(f, std::make_integer_sequence<int, N>{});
}

template <typename T>
constexpr int VEC = 16 / (int)sizeof(T);
__host__ __device__ constexpr int words_of(int values, int vec) { return (values + vec - 1) / vec; }

// 16-byte words of a record's moments up to degree D: an odd number, so the lanes' 16-byte
// reads of one word from 32 consecutive records hit distinct banks.
template <typename T, int D>
constexpr int WORDS = words_of(tri(D + 1), VEC<T>) | 1;
template <typename T, int D>
constexpr int PITCH = WORDS<T, D> * VEC<T>;

// 16 bytes of shared memory.  The read is volatile: the moments are read again for every
// pair of degrees, and a compiler that may merge those reads keeps all of them in registers
// and spills the sums (770 bytes per lane at p = 12 FP64, none this way).
template <typename T>
struct Vec;
template <>
struct Vec<double> {
    typedef double2 type;
    static __device__ __forceinline__ double get(const double2& v, int j) { return j ? v.y : v.x; }
    static __device__ __forceinline__ double2 read(unsigned address) {
        double2 v;
        asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(address));
        return v;
    }
    static __device__ __forceinline__ void write(unsigned address, int pair, double x, double y) {
        asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(address + 16 * pair), "d"(x), "d"(y));
    }
};
template <>
struct Vec<float> {
    typedef float4 type;
    static __device__ __forceinline__ float get(const float4& v, int j) {
        return j == 0 ? v.x : j == 1 ? v.y : j == 2 ? v.z : v.w;
    }
    static __device__ __forceinline__ float4 read(unsigned address) {
        float4 v;
        asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                     : "r"(address));
        return v;
    }
    static __device__ __forceinline__ void write(unsigned address, int pair, double x, double y) {
        asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(address + 8 * pair), "f"((float)x),
                     "f"((float)y));
    }
};

// 1 / (a_x! a_y!) of the coefficients in table order.
struct CartScale {
    double inv_fact2[tri(17)];
};

// The unit of length of a cell of half-width h in the mixed form: the power of two nearest h,
// so that every power and ratio of units is exact and a moment is rounded to FP32 once, where
// it is first an FP32 number, whatever the sizes of the two trees (2^-1000 to 2^1000).
__device__ __forceinline__ double unit_of(double h) {
    // the exponent, one higher from a mantissa of sqrt(2) on
    const int e = (__double2hiint(h) + (0x00100000 - 0x0006a09e)) & 0x7ff00000;
    return __hiloint2double(min(max(e, 0x01700000), 0x7e700000), 0);
}
__device__ __forceinline__ double inverse_unit(double u) {
    return __hiloint2double(0x7fe00000 - __double2hiint(u), 0);
}

// 16 bytes to shared memory, zeros without `on` (nothing is then read).
__device__ __forceinline__ void copy16(unsigned smem, const void* global, bool on) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem), "l"(global),
                 "r"(on ? 16 : 0));
}
// 8 bytes likewise.
__device__ __forceinline__ void copy8(unsigned smem, const void* global, bool on) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(smem), "l"(global),
                 "r"(on ? 8 : 0));
}
// A hint: `bytes` (a multiple of 16) from a 16-byte boundary into L2.
__device__ __forceinline__ void prefetch_l2(const void* global, int bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(global), "r"(bytes));
}
template <typename T>
constexpr bool PAIR = sizeof(T) == 4;

// One translation into the sums of degrees [B0, B1): two degrees of A at a time, advanced in
// place (even ones in e, odd ones in o), every product written out.
template <typename T, int P, int B0, int B1>
struct Products {
    static constexpr int NB = tri(B1) - tri(B0);  // coefficients b of degrees B0 .. B1 - 1
    static constexpr int NA = P - B0;             // highest moment degree they meet

    // Degree n of the Taylor coefficients A_g = A~_g / (g_x! g_y!) from degree n - 1
    // (`prev`), in place of degree n - 2 (`row`).
    template <int n>
    static __device__ __forceinline__ void advance(T* row, const T* prev, T tx, T ty, T ir2) {
        const T s = -ir2 / T(n);
        const T u = s * T(2 * n - 1) * tx, v = s * T(2 * n - 1) * ty, w = s * T(n - 1);
        static_for<n + 1>([&](auto k) {
            constexpr int gy = n - decltype(k)::value, gx = n - gy;  // from the last one down
            T x = T(0);
            if constexpr (gx >= 2 && gy >= 2) x = w * (row[gy] + row[gy - 2]);
            else if constexpr (gx >= 2) x = w * row[gy];
            else if constexpr (gy >= 2) x = w * row[gy - 2];
            if constexpr (gx >= 1) x = x + u * prev[gy];
            if constexpr (gy >= 1) x = x + v * prev[gy - 1];
            row[gy] = x;
        });
    }

    // The products of degrees n (in e; if EVEN) and n + 1 (in o; if ODD) with the moments,
    // each moment read once for both.
    template <int n, bool EVEN, bool ODD>
    static __device__ __forceinline__ void products(unsigned m, const T* e,
                                                    const T* o, int order, T* acc) {
        constexpr int top = ODD ? n + 1 : n;
        constexpr int na_max = top - B0 < NA ? top - B0 : NA;
        if constexpr (na_max >= 0) {
            T es[n + 1] = {}, os[n + 2] = {};
            if constexpr (EVEN) {
                static_for<n + 1>([&](auto k) {
                    constexpr int gy = decltype(k)::value;
                    es[gy] = e[gy] * T(factorial(n - gy) * factorial(gy));
                });
            }
            if constexpr (ODD) {  // counts up to the order only
                static_for<n + 2>([&](auto k) {
                    constexpr int gy = decltype(k)::value;
                    os[gy] = n + 1 <= order ? o[gy] * T(factorial(n + 1 - gy) * factorial(gy)) : T(0);
                });
            }
            typedef typename Vec<T>::type V;
            static_for<(tri(na_max + 1) + VEC<T> - 1) / VEC<T>>([&](auto wc) {
                constexpr int word = decltype(wc)::value;
                const V v = Vec<T>::read(m + 16 * word);
                static_for<VEC<T>>([&](auto jc) {
                    constexpr int a = word * VEC<T> + decltype(jc)::value;
                    constexpr int na = degree_of(a), ay = a - tri(na);
                    if constexpr (na <= na_max) {
                        const T ma = Vec<T>::get(v, decltype(jc)::value);
                        constexpr int be = n - na, bo = n + 1 - na;
                        if constexpr (EVEN && be >= B0 && be < B1) {
                            static_for<be + 1>([&](auto by) {
                                constexpr int y = decltype(by)::value;
                                acc[tri(be) - tri(B0) + y] += ma * es[ay + y];
                            });
                        }
                        if constexpr (ODD && bo >= B0 && bo < B1) {
                            static_for<bo + 1>([&](auto by) {
                                constexpr int y = decltype(by)::value;
                                acc[tri(bo) - tri(B0) + y] += ma * os[ay + y];
                            });
                        }
                    }
                });
            });
        }
    }

    // The products of degrees n (even, in e) and n + 1 (in o), then the next two degrees.
    template <int n>
    static __device__ __forceinline__ void step(unsigned m, T* e, T* o, T tx, T ty,
                                                T ir2, int order, T* acc) {
        if constexpr (n <= P) {
            if (n > order) return;
            if constexpr (n >= 2) advance<n>(e, o, tx, ty, ir2);
            if constexpr (n + 1 <= P) {
                if constexpr (n == 0) {
                    const T s = -ir2 * e[0];
                    o[0] = s * tx;
                    o[1] = s * ty;
                } else {
                    advance<n + 1>(o, e, tx, ty, ir2);
                }
            }
            if constexpr (n + 1 <= P && PAIR<T>) {
                products<n, true, true>(m, e, o, order, acc);
            } else {
                products<n, true, false>(m, e, o, order, acc);
                if constexpr (n + 1 <= P) {
                    if (n + 1 <= order) products<n, false, true>(m, e, o, order, acc);
                }
            }
            step<n + 2>(m, e, o, tx, ty, ir2, order, acc);
        }
    }

    // All products of one translation: t = (tx, ty), a0 = A~_0, ir2 = 1 / (t^2 + eps^2).
    static __device__ __forceinline__ void run(unsigned m, T tx, T ty, T a0, T ir2,
                                               int order, T* acc) {
        T e[P + 1], o[P + 1];
        e[0] = a0;
        // Vec::read does not tell the compiler that it reads memory: no store to the moments
        // may move past these reads, in either direction
        asm volatile("" ::: "memory");
        step<0>(m, e, o, tx, ty, ir2, order, acc);
        asm volatile("" ::: "memory");
    }
};

// A translation in FP64, in the cells' own length unit.
template <int P, int B0, int B1>
__device__ __forceinline__ void translate(const double* m, double tx, double ty, double eps2,
                                          double, double, int order, double* acc) {
    const double r2 = tx * tx + ty * ty + eps2;
    Products<double, P, B0, B1>::run(shared_address(m), tx, ty, 1.0 / sqrt(r2), 1.0 / r2, order, acc);
}

// The products of one translation times rho^(1+|b|) into the lane's moments' place (out of
// line: a rare case must not cost the others registers and instruction cache).
template <int P, int B0, int B1>
__device__ __noinline__ void far_unit_sums(float* m, float tx, float ty, float a0, float ir2,
                                           float rho, int order) {
    constexpr int NB = Products<float, P, B0, B1>::NB;
    float part[NB];
#pragma unroll
    for (int k = 0; k < NB; ++k) part[k] = 0.0f;
    Products<float, P, B0, B1>::run(shared_address(m), tx, ty, a0, ir2, order, part);
    float f = rho;
    for (int n = 0; n < B0; ++n) f *= rho;
#pragma unroll
    for (int n = B0; n < B1; ++n) {
#pragma unroll
        for (int k = tri(n); k < tri(n + 1); ++k) m[k - tri(B0)] = part[k - tri(B0)] * f;
        f *= rho;
    }
}

// A translation's own sums added to a lane's FP32 sums: one chain of roundings over the
// products of all its translations (800 at p = 12) would double the potential's error.  The
// first NC coefficients (degrees up to 2, most of the field) by Kahan's sum, its running
// errors in acc[NB ..].
template <typename T, int B0>
__host__ __device__ constexpr int compensated(int nb) {
    return sizeof(T) == 8 || B0 >= 3 ? 0 : nb < tri(3) - tri(B0) ? nb : tri(3) - tri(B0);
}
template <int NB, int NC>
__device__ __forceinline__ void add_translation(const float* part, float* acc) {
#pragma unroll
    for (int k = 0; k < NB; ++k) {
        if (k < NC) {
            const float y = part[k] - acc[NB + k], t = acc[k] + y;
            acc[NB + k] = (t - acc[k]) - y;
            acc[k] = t;
        } else {
            acc[k] += part[k];
        }
    }
}

// A translation in FP32, in the units h_s and h_d of source and destination (unit_of).  The
// record's moments are m~_a / h_s^|a| and the sums T~_b h_d^(1+|b|): with t, eps and the moments
// in units of h_d every product has the sums' unit.  The moments take (h_s / h_d)^|a| here, at
// most 16^|a|; where that grows, half of the highest power goes to A~ instead (a charge of 1e30
// times 16^16 is beyond FP32).  A source more than 16 times its destination's size (both units
// would near the ends of FP32's range) is summed in its own unit h_s and its sums multiplied by
// (h_d / h_s)^(1+|b|).
constexpr double UNIT_RANGE = 16.0;

template <int P, int B0, int B1>
__device__ __forceinline__ void translate(float* m, double tx, double ty, double eps2, double hs,
                                          double hd, int order, float* acc) {
    constexpr int NA = P - B0, NB = Products<float, P, B0, B1>::NB;
    const bool far_unit = hs > UNIT_RANGE * hd;
    const double inv = inverse_unit(far_unit ? hs : hd);
    const float x = (float)(tx * inv), y = (float)(ty * inv);
    const float r2 = (float)((double)x * x + (double)y * y + eps2 * inv * inv);
    const float ir2 = 1.0f / r2;
    float a0 = rsqrtf(r2);
    if (!far_unit) {
        if (hs != hd) {
            const float f = (float)(hs * inv);
            float p[NA + 1];
            p[0] = 1.0f;
            if (f > 1.0f) {
                const float g = 1.0f / f;
#pragma unroll
                for (int k = 0; k < NA / 2; ++k) {
                    p[0] *= g;
                    a0 *= f;
                }
            }
#pragma unroll
            for (int k = 1; k <= NA; ++k) p[k] = p[k - 1] * f;
            static_for<words_of(tri(NA + 1), 4)>([&](auto wc) {
                constexpr int a = 4 * decltype(wc)::value, last = tri(NA + 1) - 1;
                float4 v = reinterpret_cast<float4*>(m)[decltype(wc)::value];
                v.x *= p[degree_of(a)];
                v.y *= p[degree_of(a + 1 < last ? a + 1 : last)];
                v.z *= p[degree_of(a + 2 < last ? a + 2 : last)];
                v.w *= p[degree_of(a + 3 < last ? a + 3 : last)];
                reinterpret_cast<float4*>(m)[decltype(wc)::value] = v;
            });
        }
        float part[NB];
#pragma unroll
        for (int k = 0; k < NB; ++k) part[k] = 0.0f;
        Products<float, P, B0, B1>::run(shared_address(m), x, y, a0, ir2, order, part);
        add_translation<NB, compensated<float, B0>(NB)>(part, acc);
    } else {
        far_unit_sums<P, B0, B1>(m, x, y, a0, ir2, (float)(hd * inv), order);
        add_translation<NB, compensated<float, B0>(NB)>(m, acc);
    }
}

// Elements between the lanes' rows of shared memory, which hold a lane's moments (PLAIN: at
// first as they come, in FP64) and, at a row's end, its sums: an odd number of 16-byte words.
template <typename T, int P, int B0, int B1, bool PLAIN>
constexpr int STAGE_PITCH = [] {
    constexpr int sums = (words_of(Products<T, P, B0, B1>::NB, VEC<T>) | 1) * VEC<T>;
    constexpr int moments = PLAIN ? PITCH<double, P - B0> * 8 / (int)sizeof(T) : PITCH<T, P - B0>;
    return sums > moments ? sums : moments;
}();

template <typename T>
constexpr int WARPS_PER_BLOCK = 1;

// Rows [B0, B1) of degrees of the locals.  `source` holds records (td3_pack_cart_sources), or
// with PLAIN the moments themselves, copied as they are and scaled to the bits of a record by
// the lane that takes them, in every launch anew: for callers without room for records.
// PLAIN is a kernel of its own: its code on a branch of the other made that 2 to 4 % slower.
template <typename T, int P, int B0, int B1, bool PLAIN>
__global__ void __launch_bounds__(32 * WARPS_PER_BLOCK<T>)
k_m2l_cart_rows(const i64* __restrict__ row_start, const i64* __restrict__ partners, i64 n_dst,
                const double* __restrict__ dst_center, const double* __restrict__ dst_half,
                const double* __restrict__ src_center, const double* __restrict__ src_half,
                const void* __restrict__ source, int order, double eps2,
                const CartScale C, double* __restrict__ local) {
    constexpr bool MIXED = sizeof(T) == 4;
    constexpr int NB = Products<T, P, B0, B1>::NB, NA = Products<T, P, B0, B1>::NA;
    constexpr int W = WORDS<T, NA>, PITCH_S = STAGE_PITCH<T, P, B0, B1, PLAIN>;
    constexpr int Q = (NB + 3) / 4;  // coefficients a lane adds to the locals at a row's end
    extern __shared__ __align__(16) char cart_smem[];
    td3_chain_wait();
    td3_chain_release();
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, gl = lane % ROW_GL;
    T* stage = reinterpret_cast<T*>(cart_smem) + (size_t)wib * 32 * PITCH_S;
    const int n_coef = tri(order + 1);
    constexpr int NC = compensated<T, B0>(NB);
    T acc[NB + NC];
#pragma unroll
    for (int k = 0; k < NB + NC; ++k) acc[k] = T(0);

    // The moments of the lanes' partners (src < 0: none) into the lanes' rows of `stage`
    // (copies in flight until copies_done()), and the translations and sizes.
    double tx = 0.0, ty = 0.0, hs = 0.0, hd = 1.0;
    auto fetch = [&](int src, i64 d) {
        if (src >= 0) {
            // two 8-byte reads each: a caller's centres may start on any double
            tx = dst_center[2 * d] - src_center[2 * (i64)src];
            ty = dst_center[2 * d + 1] - src_center[2 * (i64)src + 1];
            if (MIXED) {
                hs = unit_of(src_half[src]);
                hd = unit_of(dst_half[d]);
            }
        }
        __syncwarp();
        if (!PLAIN) {
            // the 32 x W words in turn, 32 at a time: consecutive lanes take consecutive words
            const char* rec = static_cast<const char*>(source);
            const unsigned to = shared_address(stage);
            int p = lane / W, w = lane % W;  // record and word of this lane
#pragma unroll 8
            for (int k = 0; k < W; ++k) {
                const int s = __shfl_sync(FULL_WARP, src, p);
                copy16(to + (unsigned)(p * PITCH_S * sizeof(T)) + 16 * w,
                       rec + (size_t)(s < 0 ? 0 : s) * (16 * WORDS<T, P>) + 16 * w, s >= 0);
                p += 32 / W;
                w += 32 % W;
                if (w >= W) {
                    w -= W;
                    ++p;
                }
            }
        } else {
            // the 32 x n values in turn, 32 at a time
            const double* mom = static_cast<const double*>(source);
            const unsigned to = shared_address(stage);
            const int n = min(n_coef, tri(NA + 1));
            int p = lane / n, a = lane % n;  // record and coefficient of this lane
            const int dp = 32 / n, da = 32 % n;
#pragma unroll 4
            for (int k = 0; k < n; ++k) {
                const int s = __shfl_sync(FULL_WARP, src, p);
                copy8(to + 8u * (unsigned)(p * (PITCH_S * (int)sizeof(T) / 8) + a),
                      mom + (size_t)(s < 0 ? 0 : s) * n_coef + a, s >= 0);
                p += dp;
                a += da;
                if (a >= n) {
                    a -= n;
                    ++p;
                }
            }
        }
    };
    // The lane's plain moments as a record has them, in their place: the values written end
    // before those still to be read.  Zeros above the order: products() multiplies degree
    // order + 1 by 0, and what shared memory held may be a NaN.
    auto scale_plain = [&]() {
        const unsigned own = shared_address(stage + lane * PITCH_S);
        const double inv = MIXED ? inverse_unit(hs) : 1.0;
        double power = 1.0;  // unit^-|a|
        static_for<words_of(tri(NA + 1), 2)>([&](auto wc) {
            constexpr int pair = decltype(wc)::value;
            const double2 v = Vec<double>::read(own + 16 * pair);
            double x[2] = {0.0, 0.0};
            static_for<2>([&](auto jc) {
                constexpr int b = 2 * pair + decltype(jc)::value, nb = degree_of(b);
                if constexpr (b < tri(NA + 1)) {
                    if (MIXED && nb > 0 && b == tri(nb)) power *= inv;
                    double m = (decltype(jc)::value ? v.y : v.x) * C.inv_fact2[b];
                    if (nb & 1) m = -m;
                    if (MIXED) m *= power;
                    x[decltype(jc)::value] = b < n_coef ? m : 0.0;
                }
            });
            Vec<T>::write(own, pair, x[0], x[1]);
        });
        asm volatile("" ::: "memory");
    };
    // The group's sums through its lanes' rows of `stage` (their moments are done with):
    // lane gl ends with coefficients [first, first + Q) of all 4 lanes in sum[], added in
    // lane order.  (Exchanging halves by shuffles kept both halves of every sum live:
    // 90 FP64 sums spilled at p = 12.)
    const int first = gl * Q;
    T sum[Q];
    auto group_sums = [&](unsigned mask) {
        T* own = stage + lane * PITCH_S;
#pragma unroll
        for (int k = 0; k < NB; ++k) own[k] = k < NC ? acc[k] - acc[NB + k] : acc[k];
        __syncwarp(mask);
        const T* rows = stage + (lane & ~(ROW_GL - 1)) * PITCH_S + first;
#pragma unroll
        for (int k = 0; k < Q; ++k) {
            sum[k] = T(0);
            if (first + k < NB)
                sum[k] = (rows[k] + rows[PITCH_S + k]) + (rows[2 * PITCH_S + k] + rows[3 * PITCH_S + k]);
        }
    };
    auto add_to_locals = [&](i64 d) {
        double* out = local + d * n_coef + tri(B0) + first;
        const int count = min(NB, n_coef - tri(B0)) - first;  // this lane's coefficients
        double was[Q];
#pragma unroll
        for (int k = 0; k < Q; ++k) was[k] = k < count ? out[k] : 0.0;
        double unit = 1.0;
        int n = -1;  // the degree that `unit` = h_d^-(1 + n) belongs to
        const double inv_h = MIXED ? inverse_unit(unit_of(dst_half[d])) : 1.0;
#pragma unroll
        for (int k = 0; k < Q; ++k) {
            if (k < count) {
                const int b = first + k + tri(B0);
                double v = (double)sum[k] * C.inv_fact2[b];
                if (MIXED) {
                    while (tri(n + 1) <= b) {
                        unit *= inv_h;
                        ++n;
                    }
                    v *= unit;
                }
                out[k] = was[k] + v;
            }
        }
    };

    walk_rows(
        row_start, partners, n_dst, (i64)blockIdx.x * WARPS_PER_BLOCK<T> + wib,
        (i64)gridDim.x * WARPS_PER_BLOCK<T>, fetch,
        [&](int to_src) {
            copies_done();
            __syncwarp();
            if (PLAIN)
                scale_plain();
            else if (to_src >= 0)
                prefetch_l2(static_cast<const char*>(source) + (size_t)to_src * (16 * WORDS<T, P>),
                            16 * W);
        },
        [&]() { translate<P, B0, B1>(stage + lane * PITCH_S, tx, ty, eps2, hs, hd, order, acc); },
        [&](i64 d, bool whole, unsigned mask) {
            group_sums(mask);
            if (whole) {
#pragma unroll
                for (int k = 0; k < Q; ++k) {
                    sum[k] += __shfl_xor_sync(FULL_WARP, sum[k], 4);
                    sum[k] += __shfl_xor_sync(FULL_WARP, sum[k], 8);
                    sum[k] += __shfl_xor_sync(FULL_WARP, sum[k], 16);
                }
            }
            if (!whole || lane < ROW_GL) add_to_locals(d);
#pragma unroll
            for (int k = 0; k < NB + NC; ++k) acc[k] = T(0);
        });
}

CartScale cart_scale(int order) {
    CartScale C{};
    double f[17];
    f[0] = 1.0;
    for (int k = 1; k <= 16; ++k) f[k] = f[k - 1] * k;
    for (int n = 0; n <= order; ++n)
        for (int y = 0; y <= n; ++y) C.inv_fact2[tri(n) + y] = 1.0 / (f[n - y] * f[y]);
    return C;
}

// The templates' orders.  FP64 has 14: in the five launches of order 16's ranges, each with the
// derivatives anew, 20k particles took 1.04 ms (0.77 before the lane per translation), in three
// of its own 0.73 ms; 200k 3.34 and 2.09 ms.
int template_order(int order, bool mixed) {
    return order <= 4 ? 4 : order <= 8 ? 8 : order <= 12 ? 12 : order <= 14 && !mixed ? 14 : 16;
}

struct Args {
    const i64 *rows, *partners;
    i64 n_dst;
    const double *dst_center, *dst_half, *src_center, *src_half;
    const void* source;
    int order;
    double eps2;
    double* local;
    cudaStream_t s;
};

template <bool PLAIN, typename T, int P, int B0, int B1>
int launch_rows(const Args& a) {
    if (B0 > a.order) return TD3_OK;
    auto kernel = k_m2l_cart_rows<T, P, B0, B1, PLAIN>;
    constexpr size_t smem = sizeof(T) * 32 * STAGE_PITCH<T, P, B0, B1, PLAIN> * WARPS_PER_BLOCK<T>;
    // one resident wave of blocks, each warp an even share of the entries
    static td3_per_device blocks_of;
    int dev = 0;
    TD3_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= TD3_MAX_DEVICES) return TD3_EINVAL;
    if (!blocks_of[dev]) {
        int sms = 0, per_sm = 0;
        TD3_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)smem));
        TD3_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        TD3_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel,
                                                              32 * WARPS_PER_BLOCK<T>, smem));
        blocks_of[dev] = sms * (per_sm > 0 ? per_sm : 1);
    }
    i64 blocks = blocks_of[dev];
    const i64 most = (a.n_dst + WARPS_PER_BLOCK<T> - 1) / WARPS_PER_BLOCK<T>;
    if (blocks > most) blocks = most;
    TD3_TRY(td3_launch_chained(kernel, (unsigned)blocks, 32 * WARPS_PER_BLOCK<T>, smem, a.s, a.rows,
                               a.partners, a.n_dst, a.dst_center, a.dst_half, a.src_center,
                               a.src_half, a.source, a.order, a.eps2, cart_scale(a.order),
                               a.local));
    return TD3_OK;
}

// Consecutive ranges [B, B'), [B', B''), ... of degrees of the locals, a launch each.
template <bool PLAIN, typename T, int P, int B0, int B1, int... More>
int launch_ranges(const Args& a) {
    TD3_TRY_RC((launch_rows<PLAIN, T, P, B0, B1>(a)));
    if constexpr (sizeof...(More) > 0) return launch_ranges<PLAIN, T, P, B1, More...>(a);
    return TD3_OK;
}

// The ranges keep a launch's code near 30 KB (about 1500 products: all 1820 of p = 12 in one
// launch stall on instruction fetch, 7.0 against 5.6 ms FP64 and 8.2 against 4.4 ms FP32 for
// 12.6M translations) and the FP64 sums in registers.
template <bool PLAIN>
int launch_m2l(const Args& a, bool mixed) {
    const int p = template_order(a.order, mixed);
    if (mixed) {
        if (p == 4) return launch_ranges<PLAIN, float, 4, 0, 5>(a);
        if (p == 8) return launch_ranges<PLAIN, float, 8, 0, 9>(a);
        if (p == 12) return launch_ranges<PLAIN, float, 12, 0, 7, 13>(a);
        return launch_ranges<PLAIN, float, 16, 0, 4, 7, 11, 17>(a);
    }
    if (p == 4) return launch_ranges<PLAIN, double, 4, 0, 5>(a);
    if (p == 8) return launch_ranges<PLAIN, double, 8, 0, 9>(a);
    if (p == 12) return launch_ranges<PLAIN, double, 12, 0, 7, 13>(a);
    if (p == 14) return launch_ranges<PLAIN, double, 14, 0, 5, 10, 15>(a);
    return launch_ranges<PLAIN, double, 16, 0, 4, 7, 11, 14, 17>(a);
}

}  // namespace
