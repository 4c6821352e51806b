// The FMM of the softened Coulomb kernel in the plane with Cartesian expansions, FP64:
//   M2L by destination row  (K/cart_m2l_host/cart_m2l_host_pyccel.py:16-80)
//   L2L per level           (K/cart_downward/cart_downward_pyccel.py:14-55)
// (moments: moments.cu; L2P + P2P: nearfield.cu.)
//
// M2L (orders above 16; up to 16: cart_m2l.cuh): one warp per destination cell.  For each
// partner the warp builds the Taylor coefficients A_g(t), |g| <= p, of f = (|r|^2 + eps^2)^(-1/2) degree by degree in
// shared memory (the coefficients of one degree depend only on the two below), then
// every lane accumulates its local coefficients b over the M2L rows (b, a, a + b) of
// the reference's tables: T_b += coef * m_a * A_{a+b}.
#include "common.cuh"

namespace {

constexpr int CM2L_WARPS = 4;

__global__ void __launch_bounds__(32 * CM2L_WARPS)
k_m2l_cart(const i64* __restrict__ row_start, const i64* __restrict__ partners, i64 n_dst,
           const double* __restrict__ dst_center, const double* __restrict__ src_center,
           const double* __restrict__ moments, int order, double eps2,
           const int* __restrict__ row_a, const int* __restrict__ row_g,
           const double* __restrict__ row_coef, const int* __restrict__ b_start,
           double* __restrict__ local) {
    extern __shared__ double smem[];
    int n_coef = (order + 1) * (order + 2) / 2;
    int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    double* A = smem + (2 * wib) * n_coef;
    double* M = A + n_coef;
    constexpr int PER_LANE = 8;  // coefficients per lane held in registers
    for (i64 dst = (i64)blockIdx.x * CM2L_WARPS + wib; dst < n_dst; dst += (i64)gridDim.x * CM2L_WARPS) {
        i64 e0 = row_start[dst], e1 = row_start[dst + 1];
        if (e0 == e1) continue;
        double cx = dst_center[2 * dst], cy = dst_center[2 * dst + 1];
        for (int b0 = 0; b0 < n_coef; b0 += 32 * PER_LANE) {
            double acc[PER_LANE];
#pragma unroll
            for (int j = 0; j < PER_LANE; ++j) acc[j] = 0.0;
            for (i64 e = e0; e < e1; ++e) {
                i64 src = partners[e];
                double tx = cx - src_center[2 * src], ty = cy - src_center[2 * src + 1];
                double r2 = tx * tx + ty * ty + eps2;
                for (int i = lane; i < n_coef; i += 32) M[i] = moments[src * n_coef + i];
                if (lane == 0) A[0] = 1.0 / sqrt(r2);
                __syncwarp();
                for (int n = 1; n <= order; ++n) {
                    int base = n * (n + 1) / 2;
                    for (int b = lane; b <= n; b += 32) {
                        int a = n - b;
                        double s = 0.0;
                        if (a >= 1) s += (2 * n - 1) * tx * A[(n - 1) * n / 2 + b];
                        if (b >= 1) s += (2 * n - 1) * ty * A[(n - 1) * n / 2 + b - 1];
                        if (a >= 2) s += (n - 1) * A[(n - 2) * (n - 1) / 2 + b];
                        if (b >= 2) s += (n - 1) * A[(n - 2) * (n - 1) / 2 + b - 2];
                        A[base + b] = -s / (n * r2);
                    }
                    __syncwarp();
                }
#pragma unroll
                for (int j = 0; j < PER_LANE; ++j) {
                    int b = b0 + lane + 32 * j;
                    if (b < n_coef) {
                        double t = 0.0;
                        for (int r = b_start[b]; r < b_start[b + 1]; ++r)
                            t += row_coef[r] * M[row_a[r]] * A[row_g[r]];
                        acc[j] += t;
                    }
                }
                __syncwarp();
            }
#pragma unroll
            for (int j = 0; j < PER_LANE; ++j) {
                int b = b0 + lane + 32 * j;
                if (b < n_coef) local[dst * n_coef + b] += acc[j];
            }
        }
    }
}

// L2L of one level (orders above 16): a block per (node, child), thread b: T_b(child) += sum_g C(g, b) T_g
// s^(g-b) over the rows of b (g, d = g - b, coef).  The monomials s^d are built once per
// block into shared memory, column d_y by thread d_y as the reference's mono recurrence
// builds them (d_y factors of s_y, then s_x one at a time).
__global__ void k_l2l_cart(i64 lo, int order, int n_coef, const double* __restrict__ center,
                           const i64* __restrict__ child, const int* __restrict__ l2l_start,
                           const int* __restrict__ l2l_g, const int* __restrict__ l2l_d,
                           const double* __restrict__ l2l_coef, double* __restrict__ local) {
    extern __shared__ double shift_mono[];
    i64 node = lo + blockIdx.x / 4;
    i64 first = child[node];
    if (first < 0) return;  // the whole block: a leaf has no children
    i64 ch = first + (blockIdx.x & 3);
    double sx = center[2 * ch] - center[2 * node], sy = center[2 * ch + 1] - center[2 * node + 1];
    for (int dy = threadIdx.x; dy <= order; dy += blockDim.x) {
        double mono = 1.0;
        for (int k = 0; k < dy; ++k) mono = mono * sy;
        for (int dx = 0; dx + dy <= order; ++dx) {
            shift_mono[(dx + dy) * (dx + dy + 1) / 2 + dy] = mono;
            mono = mono * sx;
        }
    }
    __syncthreads();
    for (int b = threadIdx.x; b < n_coef; b += blockDim.x) {
        double acc = 0.0;
        for (int r = l2l_start[b]; r < l2l_start[b + 1]; ++r)
            acc += l2l_coef[r] * local[node * n_coef + l2l_g[r]] * shift_mono[l2l_d[r]];
        local[ch * n_coef + b] += acc;
    }
}

// The L2L of orders up to 16 (template order P): the shift by (s_x, s_y) as two passes of
// one-dimensional Taylor shifts (C(p + 3, 3) multiply-adds each against C(p + 4, 4) for the
// table rows: 910 against 1820 at p = 12), a thread per (child, row) with its row in
// registers.  A parent's coefficients are read once for its four children, whose rows are one
// contiguous run of the locals.  Measured (p = 12, all levels; a block per child over the
// table rows before): 2.9 -> 0.58 ms for 1M clustered particles (the locals alone move 0.1 ms),
// 0.36 -> 0.07 ms for 100k uniform ones.
template <int P>
struct CartL2L {
    static constexpr int W = P + 1, TILE = W * W;
    static constexpr int THREADS = P == 4 ? 32 : P == 16 ? 96 : 64;  // per parent, >= 4 W
    static constexpr int NODES = P == 4 ? 4 : 2;                     // parents per block, each step
};

// t_b <- sum_(g >= b) C(g, b) s^(g - b) t_g
template <int W>
__device__ __forceinline__ void taylor_shift(double (&t)[W], double s) {
#pragma unroll
    for (int i = 0; i < W - 1; ++i)
#pragma unroll
        for (int b = W - 2; b >= i; --b) t[b] += s * t[b + 1];
}

template <int P>
__global__ void __launch_bounds__(CartL2L<P>::THREADS* CartL2L<P>::NODES)
k_l2l_cart_rows(i64 lo, i64 hi, int span, int order, const double* __restrict__ center,
                const i64* __restrict__ child, double* local) {
    typedef CartL2L<P> L;
    constexpr int W = L::W, TILE = L::TILE;
    __shared__ double own[L::NODES][TILE], out[L::NODES][4][TILE];  // squares [y][x]
    __shared__ short place[W * (W + 1) / 2];  // of a coefficient in a square
    __shared__ int list[32], count;
    const int n_coef = (order + 1) * (order + 2) / 2;
    const int slot = threadIdx.x / L::THREADS, me = threadIdx.x % L::THREADS;
    for (int i = threadIdx.x; i < TILE; i += blockDim.x) {
        const int x = i % W, y = i / W;
        if (x + y <= order) place[(x + y) * (x + y + 1) / 2 + y] = (short)i;
    }
    const int k = me / W, r = me % W;  // child and row
    td3_chain_wait();
    td3_chain_release();
    const i64 first = lo + (i64)blockIdx.x * span;
    if (threadIdx.x < 32) {  // the parents among the block's cells
        const i64 node = first + threadIdx.x;
        const bool take = (int)threadIdx.x < span && node < hi && child[node] >= 0;
        const unsigned m = __ballot_sync(0xffffffffu, take);
        if (take) list[__popc(m & ((1u << threadIdx.x) - 1u))] = threadIdx.x;
        if (threadIdx.x == 0) count = __popc(m);
    }
    __syncthreads();
    for (int base = 0; base < count; base += L::NODES) {
        const bool live = base + slot < count;
        const i64 node = first + list[live ? base + slot : base];
        const i64 kids = child[node];
        if (live) {
            for (int c = me; c < n_coef; c += L::THREADS)
                own[slot][place[c]] = local[node * n_coef + c];
        }
        __syncthreads();
        const bool work = live && k < 4 && r <= order;
        double t[W];
        if (work) {  // row (., r) along x
            const double s = center[2 * (kids + k)] - center[2 * node];
#pragma unroll
            for (int x = 0; x < W; ++x) t[x] = x + r <= order ? own[slot][r * W + x] : 0.0;
            taylor_shift<W>(t, s);
#pragma unroll
            for (int x = 0; x < W; ++x) out[slot][k][r * W + x] = t[x];
        }
        __syncthreads();
        if (work) {  // row (r, .) along y
            const double s = center[2 * (kids + k) + 1] - center[2 * node + 1];
#pragma unroll
            for (int y = 0; y < W; ++y) t[y] = y + r <= order ? out[slot][k][y * W + r] : 0.0;
            taylor_shift<W>(t, s);
#pragma unroll
            for (int y = 0; y < W; ++y) out[slot][k][y * W + r] = t[y];
        }
        __syncthreads();
        if (live) {
            double* to = local + kids * n_coef;
            for (int c = me; c < n_coef; c += L::THREADS) {
#pragma unroll
                for (int kid = 0; kid < 4; ++kid) to[kid * n_coef + c] += out[slot][kid][place[c]];
            }
        }
        __syncthreads();
    }
}

template <int P>
int launch_l2l_rows(const i64* levels, i64 n_levels, int order, const double* center,
                    const i64* child, double* local, cudaStream_t s) {
    for (i64 level = 0; level + 1 < n_levels; ++level) {
        const i64 lo = levels[level], hi = levels[level + 1];
        if (hi <= lo) continue;
        // consecutive cells a block picks its parents from: a few blocks per SM, 32 at most
        const i64 pick = (hi - lo) / (148 * 8);
        const int span = pick < CartL2L<P>::NODES ? CartL2L<P>::NODES : pick > 32 ? 32 : (int)pick;
        TD3_TRY(td3_launch_chained(k_l2l_cart_rows<P>, td3_blocks(hi - lo, span),
                                   CartL2L<P>::THREADS * CartL2L<P>::NODES, 0, s, lo, hi, span,
                                   order, center, child, local));
    }
    return TD3_OK;
}

}  // namespace

extern "C" int td3_cart_m2l(const int64_t* row_start, const int64_t* partners, int64_t n_dst,
                            const double* dst_center, const double* src_center,
                            const double* moments, int order, double softening,
                            const int* row_a, const int* row_g, const double* row_coef,
                            const int* b_start, double* local, void* stream) {
    if (n_dst < 0 || order < 0 || order > TD3_MAX_ORDER) return TD3_EINVAL;
    if (n_dst == 0) return TD3_OK;
    cudaStream_t s = td3_stream(stream);
    int n_coef = (order + 1) * (order + 2) / 2;
    if (order <= 16)
        return td3_cart_m2l_unpacked(row_start, partners, n_dst, dst_center, nullptr, src_center,
                                     nullptr, moments, order, softening, false, local, s);
    size_t smem = sizeof(double) * 2 * n_coef * CM2L_WARPS;
    if (smem > 48 * 1024)
        TD3_TRY(cudaFuncSetAttribute(k_m2l_cart, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)smem));
    i64 blocks = (n_dst + CM2L_WARPS - 1) / CM2L_WARPS;
    if (blocks > 148 * 64) blocks = 148 * 64;
    k_m2l_cart<<<(unsigned)blocks, 32 * CM2L_WARPS, smem, s>>>(
        row_start, partners, n_dst, dst_center, src_center, moments, order,
        softening * softening, row_a, row_g, row_coef, b_start, local);
    TD3_CHECK_LAUNCH();
    return TD3_OK;
}

extern "C" int td3_cart_downward(const int64_t* levels, int64_t n_levels, const double* node_center,
                                 const int64_t* node_child, int order, const int64_t* ex,
                                 const int64_t* ey, const int* l2l_start, const int* l2l_g,
                                 const int* l2l_d, const double* l2l_coef, double* local,
                                 void* stream) {
    if (n_levels < 1 || order < 0 || order > TD3_MAX_ORDER) return TD3_EINVAL;
    cudaStream_t s = td3_stream(stream);
    if (order <= 4) return launch_l2l_rows<4>(levels, n_levels, order, node_center, node_child, local, s);
    if (order <= 8) return launch_l2l_rows<8>(levels, n_levels, order, node_center, node_child, local, s);
    if (order <= 12) return launch_l2l_rows<12>(levels, n_levels, order, node_center, node_child, local, s);
    if (order <= 16) return launch_l2l_rows<16>(levels, n_levels, order, node_center, node_child, local, s);
    int n_coef = (order + 1) * (order + 2) / 2;
    unsigned threads = (unsigned)((n_coef + 31) / 32 * 32);
    if (threads > 256) threads = 256;
    size_t smem = sizeof(double) * n_coef;
    if (smem > 48 * 1024)
        TD3_TRY(cudaFuncSetAttribute(k_l2l_cart, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)smem));
    (void)ex;
    (void)ey;
    for (i64 level = 0; level + 1 < n_levels; ++level) {
        i64 lo = levels[level], hi = levels[level + 1];
        if (hi <= lo) continue;
        k_l2l_cart<<<(unsigned)(4 * (hi - lo)), threads, smem, s>>>(
            lo, order, n_coef, node_center, node_child, l2l_start, l2l_g, l2l_d, l2l_coef, local);
    }
    TD3_CHECK_LAUNCH();
    return TD3_OK;
}

extern "C" int td3_cart_m2l_mixed(const int64_t* row_start, const int64_t* partners,
                                  int64_t n_dst, const double* dst_center,
                                  const double* dst_half, const double* src_center,
                                  const double* src_half, const double* moments, int order,
                                  double softening, double* local, void* stream) {
    if (n_dst < 0 || order < 0 || order > 16) return TD3_EINVAL;
    if (n_dst == 0) return TD3_OK;
    return td3_cart_m2l_unpacked(row_start, partners, n_dst, dst_center, dst_half, src_center,
                                 src_half, moments, order, softening, true, local,
                                 td3_stream(stream));
}
