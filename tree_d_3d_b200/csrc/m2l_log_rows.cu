// FP64 M2L of the log kernel for orders up to 20, a lane per translation
// (K/fmm_m2l_host/fmm_m2l_host_pyccel.py:16-105; higher orders: fmm_log.cu).
//
// b_l += +-w^l sum_k C[k, l] a_k w^k, w = 1 / t: a lane takes one translation whole, with the
// scaled moments and the destination's sums in registers, so that the 2 (p + 1)^2
// multiply-adds of the real matrix product are all there is on the FP64 pipe.  The moments
// come through shared memory (copied by the warp, 8 bytes per lane, coalesced), the matrix
// is read there too, two values by one broadcast for four multiply-adds.  Rows as walk_rows.
//
// Measured (theta 0.5; a group of 16 or 32 lanes per translation, a lane per coefficient and
// both factors in shared memory before): 1M clustered particles, 12.6M translations, p = 8 /
// 12 / 16 / 20: 3.06 / 3.28 / 8.08 / 8.54 -> 1.1 / 1.58 / 2.5 / 3.7 ms; 200k, p = 12: 0.69 ->
// 0.41 ms; 5000, p = 12: 0.060 -> 0.037 ms.
#include "row_groups.cuh"

namespace {

// 8 bytes to shared memory, zero without `on` (nothing is then read).
__device__ __forceinline__ void copy8(unsigned smem, const double* global, bool on) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(smem), "l"(global),
                 "r"(on ? 8 : 0));
}

// Warps per SM that the registers are held to: to order 8 16 (200k, p = 8: 0.23 against 0.28
// ms), to order 12 12; above, the sums and moments want all of a lane's (10 warps at p = 14:
// 0.54 against 0.45 ms).
template <int P>
__global__ void __launch_bounds__(32, P <= 8 ? 16 : P <= 12 ? 12 : 1)
k_m2l_log_rows(const i64* __restrict__ row_start, const i64* __restrict__ partners, i64 n_dst,
               const double* __restrict__ dst_center, const double* __restrict__ src_center,
               const double* __restrict__ moment_re, const double* __restrict__ moment_im,
               int order, const double* __restrict__ coeff, double* __restrict__ local_re,
               double* __restrict__ local_im) {
    constexpr int W = P + 1, WE = (W + 1) & ~1;  // WE: a matrix row, whole 16-byte words
    constexpr int PITCH = 2 * W + 1;             // a lane's moments, real then imaginary parts
    constexpr int Q = (W + ROW_GL - 1) / ROW_GL;
    __shared__ __align__(16) double matrix[W][WE];  // [l][k]
    __shared__ double stage[32 * PITCH];
    td3_chain_wait();
    td3_chain_release();
    const int lane = threadIdx.x, gl = lane % ROW_GL, w = order + 1;
    for (int i = lane; i < W * WE; i += 32) {
        const int l = i / WE, k = i % WE;
        matrix[l][k] = l < w && k < w ? coeff[k * w + l] : 0.0;
    }
    __syncwarp();
    double br[W], bi[W];
#pragma unroll
    for (int l = 0; l < W; ++l) br[l] = bi[l] = 0.0;
    double* own = stage + lane * PITCH;
    double tx = 0.0, ty = 0.0;

    auto fetch = [&](int src, i64 d) {
        if (src >= 0) {
            // two 8-byte reads each: a caller's centres may start on any double
            tx = dst_center[2 * d] - src_center[2 * (i64)src];
            ty = dst_center[2 * d + 1] - src_center[2 * (i64)src + 1];
        }
        __syncwarp();
        // the 32 x 2 w values in turn, 32 at a time
        const int n = 2 * w;
        const unsigned to = shared_address(stage);
        int p = lane / n, j = lane % n;  // record and value of this lane
        const int dp = 32 / n, dj = 32 % n;
#pragma unroll 4
        for (int k = 0; k < n; ++k) {
            const int s = __shfl_sync(FULL_WARP, src, p);
            const i64 at = (i64)(s < 0 ? 0 : s) * w;
            const bool im = j >= w;
            copy8(to + 8u * (unsigned)(p * PITCH + (im ? W + j - w : j)),
                  im ? moment_im + at + (j - w) : moment_re + at + j, s >= 0);
            p += dp;
            j += dj;
            if (j >= n) {
                j -= n;
                ++p;
            }
        }
    };
    auto translate = [&]() {
        const double t2 = tx * tx + ty * ty, inv = 1.0 / t2;
        const double wr = tx * inv, wi = -ty * inv;
        double ar[W], ai[W];
        double pr = 1.0, pi = 0.0;
#pragma unroll
        for (int k = 0; k < W; ++k) {
            const double xr = own[k], xi = own[W + k];
            // above the order: zero by selection (the place is not written, and w^k may be
            // infinite where w^order is not)
            ar[k] = k < w ? xr * pr - xi * pi : 0.0;
            ai[k] = k < w ? xr * pi + xi * pr : 0.0;
            const double nr = pr * wr - pi * wi;
            pi = pr * wi + pi * wr;
            pr = nr;
        }
        // only Re ln t = ln |t| reaches phi and E
        const double ln = 0.5 * log(t2);
        br[0] += ar[0] * ln;
        bi[0] += ai[0] * ln;
        double qr = -1.0, qi = 0.0;  // -(-1)^l w^l
#pragma unroll
        for (int l = 0; l < W; ++l) {
            double sr = 0.0, si = 0.0;
#pragma unroll
            for (int k = 0; k < W; k += 2) {
                const double2 c = *reinterpret_cast<const double2*>(&matrix[l][k]);
                sr += c.x * ar[k];
                si += c.x * ai[k];
                if (k + 1 < W) {
                    sr += c.y * ar[k + 1];
                    si += c.y * ai[k + 1];
                }
            }
            if (l == 0) {
                br[0] -= sr;
                bi[0] -= si;
            } else {
                br[l] += sr * qr - si * qi;
                bi[l] += sr * qi + si * qr;
            }
            const double nr = qi * wi - qr * wr;
            qi = -(qr * wi + qi * wr);
            qr = nr;
        }
    };
    auto finish = [&](i64 d, bool whole, unsigned mask) {
        // the group's sums through its lanes' places (their moments are done with)
#pragma unroll
        for (int l = 0; l < W; ++l) {
            own[l] = br[l];
            own[W + l] = bi[l];
            br[l] = bi[l] = 0.0;
        }
        __syncwarp(mask);
        const double* rows = stage + (lane & ~(ROW_GL - 1)) * PITCH;
#pragma unroll
        for (int j = 0; j < Q; ++j) {
            const int l = gl + ROW_GL * j;
            double r = 0.0, i = 0.0;
            if (l < W) {
                r = (rows[l] + rows[PITCH + l]) + (rows[2 * PITCH + l] + rows[3 * PITCH + l]);
                const double* im = rows + W + l;
                i = (im[0] + im[PITCH]) + (im[2 * PITCH] + im[3 * PITCH]);
            }
            if (whole) {
#pragma unroll
                for (int o = ROW_GL; o < 32; o <<= 1) {
                    r += __shfl_xor_sync(FULL_WARP, r, o);
                    i += __shfl_xor_sync(FULL_WARP, i, o);
                }
            }
            if (l < w && (!whole || lane < ROW_GL)) {
                local_re[d * w + l] += r;
                local_im[d * w + l] += i;
            }
        }
    };
    walk_rows(
        row_start, partners, n_dst, blockIdx.x, gridDim.x, fetch,
        [&](int) {
            copies_done();
            __syncwarp();
        },
        translate, finish);
}

template <int P>
int launch_rows(const i64* row_start, const i64* partners, i64 n_dst, const double* dst_center,
                const double* src_center, const double* mre, const double* mim, int order,
                const double* coeff, double* lre, double* lim, cudaStream_t s) {
    auto kernel = k_m2l_log_rows<P>;
    // one resident wave of one-warp blocks, each an even share of the entries
    static td3_per_device blocks_of;
    int dev = 0;
    TD3_TRY(cudaGetDevice(&dev));
    if (dev < 0 || dev >= TD3_MAX_DEVICES) return TD3_EINVAL;
    if (!blocks_of[dev]) {
        int sms = 0, per_sm = 0;
        TD3_TRY(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                     cudaSharedmemCarveoutMaxShared));
        TD3_TRY(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
        TD3_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 32, 0));
        blocks_of[dev] = sms * (per_sm > 0 ? per_sm : 1);
    }
    i64 blocks = blocks_of[dev];
    if (blocks > n_dst) blocks = n_dst;
    TD3_TRY(td3_launch_chained(kernel, (unsigned)blocks, 32, 0, s, row_start, partners, n_dst,
                               dst_center, src_center, mre, mim, order, coeff, lre, lim));
    return TD3_OK;
}

}  // namespace

int td3_m2l_log_rows(const i64* row_start, const i64* partners, i64 n_dst,
                     const double* dst_center, const double* src_center, const double* moment_re,
                     const double* moment_im, int order, const double* coeff, double* local_re,
                     double* local_im, cudaStream_t s) {
#define TD3_ROWS(P)                                                                          \
    if (order <= P)                                                                          \
    return launch_rows<P>(row_start, partners, n_dst, dst_center, src_center, moment_re,     \
                          moment_im, order, coeff, local_re, local_im, s)
    TD3_ROWS(4);
    TD3_ROWS(8);
    TD3_ROWS(10);
    TD3_ROWS(12);
    TD3_ROWS(14);
    TD3_ROWS(16);
    TD3_ROWS(18);
    TD3_ROWS(20);
#undef TD3_ROWS
    return TD3_EINVAL;
}
