// The elementwise parts of one ElectrostaticSimulation step (src/tree_d_3d/simulation.py:
// 800-835), a launch each, and what its host logic wants to know of the state, three launches
// and one host read: a step of 1000 particles by separate array operations took 129 launches
// and 12 host reads, 1.15 ms for 0.12 ms of pair sums; now ten of the library's, a dozen of
// torch's and three reads, 0.29 ms.
#include "common.cuh"

namespace {

constexpr int SIM_THREADS = 256;

struct Walls {
    int count;
    int axis[4];
    double sign[4], value[4];
};

// Facts of the state, as td3_sim_scan documents them.  The four bounds are kept as unsigned
// integers that order as the doubles do, so that blocks combine them by atomics.
struct Facts {
    unsigned long long low[2], high[2];
    unsigned long long not_finite, charged, fixed, changed, outside;
};

__device__ __forceinline__ unsigned long long ordered(double v) {
    const unsigned long long b = (unsigned long long)__double_as_longlong(v);
    return b >> 63 ? ~b : b | 0x8000000000000000ull;
}

__global__ void k_sim_facts_init(Facts* f) {
    f->low[0] = f->low[1] = ~0ull;
    f->high[0] = f->high[1] = 0ull;
    f->not_finite = f->charged = f->fixed = f->changed = f->outside = 0;
}

__global__ void __launch_bounds__(SIM_THREADS)
k_sim_scan(const double* __restrict__ pos, const double* __restrict__ charge,
           const unsigned char* __restrict__ fixed, i64 n, const double* __restrict__ last_pos,
           const double* __restrict__ last_charge, const unsigned char* __restrict__ last_fixed,
           const Walls walls, Facts* facts) {
    unsigned long long lo[2] = {~0ull, ~0ull}, hi[2] = {0, 0};
    unsigned count[5] = {0, 0, 0, 0, 0};  // not finite, charged, fixed, changed, outside
    for (i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (i64)gridDim.x * blockDim.x) {
        const double p[2] = {pos[i], pos[n + i]}, q = charge[i];
        const bool fx = fixed[i] != 0;
        count[0] += !isfinite(p[0]) || !isfinite(p[1]);
        count[1] += q != 0.0;
        count[2] += fx;
        if (last_pos)
            count[3] += !(p[0] == last_pos[i] && p[1] == last_pos[n + i] && q == last_charge[i] &&
                          fx == (last_fixed[i] != 0));
        bool out = false;
        for (int w = 0; w < walls.count; ++w)
            out |= walls.sign[w] * (p[walls.axis[w]] - walls.value[w]) > 0.0;
        count[4] += out;
#pragma unroll
        for (int a = 0; a < 2; ++a) {
            const unsigned long long v = ordered(p[a]);
            lo[a] = v < lo[a] ? v : lo[a];
            hi[a] = v > hi[a] ? v : hi[a];
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
        for (int a = 0; a < 2; ++a) {
            const unsigned long long l = __shfl_xor_sync(0xffffffffu, lo[a], o);
            const unsigned long long h = __shfl_xor_sync(0xffffffffu, hi[a], o);
            lo[a] = l < lo[a] ? l : lo[a];
            hi[a] = h > hi[a] ? h : hi[a];
        }
    }
#pragma unroll
    for (int c = 0; c < 5; ++c) count[c] = __reduce_add_sync(0xffffffffu, count[c]);
    if (threadIdx.x & 31) return;
    for (int a = 0; a < 2; ++a) {
        atomicMin(&facts->low[a], lo[a]);
        atomicMax(&facts->high[a], hi[a]);
    }
    unsigned long long* to = &facts->not_finite;
    for (int c = 0; c < 5; ++c)
        if (count[c]) atomicAdd(to + c, (unsigned long long)count[c]);
}

// The bounds back to doubles, the counts to whole doubles.
__global__ void k_sim_facts_out(const Facts* f, double* out) {
    const int t = threadIdx.x;
    if (t < 4) {
        const unsigned long long b = t & 1 ? f->high[t >> 1] : f->low[t >> 1];
        out[t] = __longlong_as_double((long long)(b >> 63 ? b & 0x7fffffffffffffffull : ~b));
    } else if (t < 9) {
        out[t] = (double)(&f->not_finite)[t - 4];
    }
}

// Half kick by the electric force, then the exact drift of a uniform B_z over dt: a =
// sinc(angle), b = angle / 2 sinc(angle / 2)^2 with angle = q B_z dt / m.
__global__ void k_sim_kick_drift(const double* __restrict__ pos, const double* __restrict__ vel,
                                 const double* __restrict__ electric,
                                 const double* __restrict__ charge, const double* __restrict__ mass,
                                 const unsigned char* __restrict__ fixed, i64 n, double dt,
                                 double b_z, double* __restrict__ new_pos,
                                 double* __restrict__ new_vel) {
    const i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double mobile = fixed[i] ? 0.0 : 1.0, m = mass[i], angle = charge[i] / m * b_z * dt;
    const double vx = vel[i] + 0.5 * dt * electric[i] / m * mobile;
    const double vy = vel[n + i] + 0.5 * dt * electric[n + i] / m * mobile;
    double s, c;
    sincos(angle, &s, &c);
    const double half = 0.5 * angle, sh = half == 0.0 ? 1.0 : sin(half) / half;
    const double a = angle == 0.0 ? 1.0 : s / angle, b = half * (sh * sh);
    new_pos[i] = pos[i] + dt * (a * vx + b * vy) * mobile;
    new_pos[n + i] = pos[n + i] + dt * (a * vy - b * vx) * mobile;
    new_vel[i] = mobile != 0.0 ? c * vx + s * vy : vx;
    new_vel[n + i] = mobile != 0.0 ? c * vy - s * vx : vy;
}

// The second half kick and the total force q (E + v x B).
__global__ void k_sim_kick_force(const double* __restrict__ vel, const double* __restrict__ electric,
                                 const double* __restrict__ charge, const double* __restrict__ mass,
                                 const unsigned char* __restrict__ fixed, i64 n, double dt,
                                 double b_z, double* __restrict__ new_vel,
                                 double* __restrict__ force) {
    const i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double mobile = fixed[i] ? 0.0 : 1.0, m = mass[i], qb = charge[i] * b_z;
    const double vx = vel[i] + 0.5 * dt * electric[i] / m * mobile;
    const double vy = vel[n + i] + 0.5 * dt * electric[n + i] / m * mobile;
    new_vel[i] = vx;
    new_vel[n + i] = vy;
    force[i] = electric[i] + qb * vy;
    force[n + i] = electric[n + i] + qb * -vx;
}

}  // namespace

extern "C" size_t td3_sim_scan_workspace_size(void) { return td3_ws_bytes<Facts>(1); }

extern "C" int td3_sim_scan(const double* pos, const double* charge, const uint8_t* fixed, int64_t n,
                            const double* last_pos, const double* last_charge,
                            const uint8_t* last_fixed, int n_walls, const int* wall_axis,
                            const double* wall_sign, const double* wall_value, double* facts,
                            void* workspace, size_t workspace_bytes, void* stream) {
    if (n < 0 || n_walls < 0 || n_walls > 4) return TD3_EINVAL;
    if (workspace_bytes < sizeof(Facts)) return TD3_EWORKSPACE;
    Walls walls{n_walls, {}, {}, {}};
    for (int w = 0; w < n_walls; ++w) {
        if (wall_axis[w] != 0 && wall_axis[w] != 1) return TD3_EINVAL;
        walls.axis[w] = wall_axis[w];
        walls.sign[w] = wall_sign[w];
        walls.value[w] = wall_value[w];
    }
    cudaStream_t s = td3_stream(stream);
    Facts* f = static_cast<Facts*>(workspace);
    k_sim_facts_init<<<1, 1, 0, s>>>(f);
    if (n) {
        unsigned blocks = td3_blocks(n, SIM_THREADS);
        if (blocks > 148 * 4) blocks = 148 * 4;
        k_sim_scan<<<blocks, SIM_THREADS, 0, s>>>(pos, charge, fixed, n, last_pos, last_charge,
                                                  last_fixed, walls, f);
    }
    k_sim_facts_out<<<1, 32, 0, s>>>(f, facts);
    TD3_CHECK_LAUNCH();
    return TD3_OK;
}

extern "C" int td3_sim_kick_drift(const double* pos, const double* vel, const double* electric,
                                  const double* charge, const double* mass, const uint8_t* fixed,
                                  int64_t n, double dt, double b_z, double* new_pos,
                                  double* new_vel, void* stream) {
    if (n < 0) return TD3_EINVAL;
    if (n == 0) return TD3_OK;
    k_sim_kick_drift<<<td3_blocks(n, SIM_THREADS), SIM_THREADS, 0, td3_stream(stream)>>>(
        pos, vel, electric, charge, mass, fixed, n, dt, b_z, new_pos, new_vel);
    TD3_CHECK_LAUNCH();
    return TD3_OK;
}

extern "C" int td3_sim_kick_force(const double* vel, const double* electric, const double* charge,
                                  const double* mass, const uint8_t* fixed, int64_t n, double dt,
                                  double b_z, double* new_vel, double* force, void* stream) {
    if (n < 0) return TD3_EINVAL;
    if (n == 0) return TD3_OK;
    k_sim_kick_force<<<td3_blocks(n, SIM_THREADS), SIM_THREADS, 0, td3_stream(stream)>>>(
        vel, electric, charge, mass, fixed, n, dt, b_z, new_vel, force);
    TD3_CHECK_LAUNCH();
    return TD3_OK;
}
