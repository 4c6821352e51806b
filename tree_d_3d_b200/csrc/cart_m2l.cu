// The Cartesian M2L of orders up to 16 from records of the source cells, and those records
// (cart_m2l.cuh).
#include "cart_m2l.cuh"

namespace {

// Records for the M2L: m~_a (FP64), or m~_a / unit^|a| (FP32); zero beyond the order.
template <typename T, int P>
__global__ void k_pack_cart(i64 count, int order, const double* __restrict__ moments,
                            const double* __restrict__ half, const CartScale C,
                            T* __restrict__ rec) {
    constexpr int N = PITCH<T, P>;
    td3_chain_wait();
    td3_chain_release();
    const int n_coef = tri(order + 1);
    const i64 total = count * N;
    for (i64 t = (i64)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (i64)gridDim.x * blockDim.x) {
        const i64 node = t / N;
        const int a = (int)(t - node * N);
        double v = 0.0;
        if (a < n_coef) {
            const int na = degree_of(a);
            v = moments[node * n_coef + a] * C.inv_fact2[a];
            if (na & 1) v = -v;
            if (sizeof(T) == 4) {
                const double inv_h = inverse_unit(unit_of(half[node]));
                for (int k = 0; k < na; ++k) v *= inv_h;
            }
        }
        rec[t] = (T)v;
    }
}

template <typename T, int P>
int launch_pack(i64 count, int order, const double* moments, const double* half, void* rec,
                cudaStream_t s) {
    TD3_TRY(td3_launch_chained(k_pack_cart<T, P>, min(td3_blocks(count * PITCH<T, P>, 256), 148u * 32u),
                               256, 0, s, count, order, moments, half, cart_scale(order),
                               static_cast<T*>(rec)));
    return TD3_OK;
}

}  // namespace

extern "C" int td3_cart_record_bytes(int order, int mixed) {
    if (order < 0 || order > 16) return TD3_EINVAL;
    switch (template_order(order, mixed != 0)) {
        case 4: return 16 * (mixed ? WORDS<float, 4> : WORDS<double, 4>);
        case 8: return 16 * (mixed ? WORDS<float, 8> : WORDS<double, 8>);
        case 12: return 16 * (mixed ? WORDS<float, 12> : WORDS<double, 12>);
        case 14: return 16 * WORDS<double, 14>;
        default: return 16 * (mixed ? WORDS<float, 16> : WORDS<double, 16>);
    }
}

extern "C" int td3_pack_cart_sources(int64_t count, int order, const double* moments,
                                     const double* node_half, int mixed, void* records,
                                     void* stream) {
    if (count < 0 || order < 0 || order > 16) return TD3_EINVAL;
    if (count == 0) return TD3_OK;
    cudaStream_t s = td3_stream(stream);
    switch (template_order(order, mixed != 0)) {
        case 4:
            return mixed ? launch_pack<float, 4>(count, order, moments, node_half, records, s)
                         : launch_pack<double, 4>(count, order, moments, node_half, records, s);
        case 8:
            return mixed ? launch_pack<float, 8>(count, order, moments, node_half, records, s)
                         : launch_pack<double, 8>(count, order, moments, node_half, records, s);
        case 12:
            return mixed ? launch_pack<float, 12>(count, order, moments, node_half, records, s)
                         : launch_pack<double, 12>(count, order, moments, node_half, records, s);
        case 14: return launch_pack<double, 14>(count, order, moments, node_half, records, s);
        default:
            return mixed ? launch_pack<float, 16>(count, order, moments, node_half, records, s)
                         : launch_pack<double, 16>(count, order, moments, node_half, records, s);
    }
}

extern "C" int td3_cart_m2l_rows(const int64_t* row_start, const int64_t* partners, int64_t n_dst,
                                 const double* dst_center, const double* dst_half,
                                 const double* src_center, const double* src_half,
                                 const void* records, int order, double softening, int mixed,
                                 double* local, void* stream) {
    if (n_dst < 0 || order < 0 || order > 16) return TD3_EINVAL;
    if (n_dst == 0) return TD3_OK;
    const Args a{row_start, partners, n_dst, dst_center, dst_half,
                 src_center, src_half, records, order, softening * softening, local,
                 td3_stream(stream)};
    return launch_m2l<false>(a, mixed != 0);
}
