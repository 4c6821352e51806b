// The Cartesian M2L of orders up to 16 from the moments themselves (cart_m2l.cuh), behind
// fmm_cart.cu's entry points.  Nothing in this package calls it for those orders.
//
// Milliseconds for 12.6M translations (1M clustered particles, theta 0.5), FP64 / FP32 at
// p = 4, 8, 12 and 16: a lane per coefficient run, without records, 2.5 / 2.7, 7.1 / 6.1,
// 18.6 / 13.2, 57 / 33; this way 0.62 / 0.66, 2.2 / 2.5, 9.1 / 9.4, 28 / 30.
#include "cart_m2l.cuh"

int td3_cart_m2l_unpacked(const i64* row_start, const i64* partners, i64 n_dst,
                          const double* dst_center, const double* dst_half,
                          const double* src_center, const double* src_half,
                          const double* moments, int order, double softening, bool mixed,
                          double* local, cudaStream_t s) {
    const Args a{row_start, partners, n_dst, dst_center, dst_half,
                 src_center, src_half, moments, order, softening * softening, local, s};
    return launch_m2l<true>(a, mixed);
}

