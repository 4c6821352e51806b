// Interaction lists of the FMM:
//   fmm_traverse   mutual dual-tree traversal from (root, root), generation by
//                  generation (K/fmm_traverse/fmm_traverse_pyccel.py:15-106, driven by
//                  FlatQuadtree._traverse, ft:1318-1358);
//   dual_traverse  one-way traversal of a target tree against a source tree
//                  (K/dual_traverse/dual_traverse_pyccel.py:14-86);
//   pair_csr       pair lists as rows by node (K/pair_csr/pair_csr_pyccel.py:12-45).
//
// A generation classifies every frontier pair (M2L, P2P, its 4 or 10 child pairs, or
// dropped) and writes each output to its slot in one launch: the tiles of the frontier get
// their first slots from the tiles before them (decoupled look-back), so the lists come out
// in the reference's serial order.  The frontier sizes stay on the device; the host looks at
// them every few generations.  The
// predicates use exactly rounded operations (this file is compiled with --fmad=false).
#include "common.cuh"

namespace {

constexpr int TRAV_THREADS = 256;

struct Pair {
    i64 a, b;
};

// A frontier pair: node indices fit 32 bits (the entry points check the node counts).
struct __align__(8) FPair {
    int a, b;
};

enum : int { ACT_NONE = 0, ACT_M2L = 1, ACT_P2P = 2, ACT_SELF = 3, ACT_SPLIT_A = 4, ACT_SPLIT_B = 5 };

// A node as the traversal reads it: one 32-byte record (one memory sector) instead of
// five arrays.  child is the first child (-1 for a leaf), filled is 0 for an empty cell.
struct __align__(32) NodeRec {
    double cx, cy, half;
    int child, filled;
};

__global__ void k_node_records(i64 count, const double* __restrict__ center,
                               const double* __restrict__ half, const i64* __restrict__ start,
                               const i64* __restrict__ end, const i64* __restrict__ child,
                               NodeRec* __restrict__ rec) {
    td3_chain_wait();
    td3_chain_release();
    i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    rec[i] = NodeRec{center[2 * i], center[2 * i + 1], half[i], (int)child[i],
                     end[i] != start[i] ? 1 : 0};
}

// The decision of the mutual traversal for pair (a, b) (fmm_traverse_pyccel.py:48-106).
__device__ __forceinline__ int classify_mutual(i64 a, i64 b, const NodeRec* __restrict__ rec,
                                               double theta) {
    NodeRec ra = rec[a], rb = rec[b];
    if (!ra.filled || !rb.filled) return ACT_NONE;
    bool leaf_a = ra.child < 0, leaf_b = rb.child < 0;
    if (a == b) return leaf_a ? ACT_P2P : ACT_SELF;
    double dx = xsub(ra.cx, rb.cx);
    double dy = xsub(ra.cy, rb.cy);
    double distance = xsqrt(xnorm2(dx, dy));
    double radii = xmul(TD3_ROOT2, xadd(ra.half, rb.half));
    if (radii < xmul(theta, distance)) return ACT_M2L;
    if (leaf_a && leaf_b) return ACT_P2P;
    if (leaf_b || (!leaf_a && ra.half >= rb.half)) return ACT_SPLIT_A;
    return ACT_SPLIT_B;
}

// The one-way decision for (target cell a, source cell b) (dual_traverse_pyccel.py:46-86).
__device__ __forceinline__ int classify_dual(i64 a, i64 b, const NodeRec* __restrict__ t_rec,
                                             const NodeRec* __restrict__ s_rec, double theta) {
    NodeRec ra = t_rec[a], rb = s_rec[b];
    if (!ra.filled || !rb.filled) return ACT_NONE;
    double dx = xsub(ra.cx, rb.cx);
    double dy = xsub(ra.cy, rb.cy);
    if (xmul(TD3_ROOT2, xadd(ra.half, rb.half)) < xmul(theta, xsqrt(xnorm2(dx, dy))))
        return ACT_M2L;
    bool leaf_a = ra.child < 0, leaf_b = rb.child < 0;
    if (leaf_a && leaf_b) return ACT_P2P;
    if (leaf_b || (!leaf_a && ra.half >= rb.half)) return ACT_SPLIT_A;
    return ACT_SPLIT_B;
}

// ------------------------------------------------------------------ generations
// A generation is one launch that reads the frontier size from device memory.  Its blocks
// take tiles of GEN_TILE pairs in order (a ticket each); a tile's pairs are classified once,
// with their actions in registers, its counts published, and its first slots found from the
// tiles before it: their counts up to the nearest one whose own first slots are known
// (Merrill and Garland's decoupled look-back).  Tiles are taken in order by resident blocks,
// so a tile's predecessors are always under way; the wait for them is bounded all the same
// (LOOK_LIMIT polls, then the state's `failed`, which the host turns into an error).  One
// thread reads for its block what the other blocks may write meanwhile (`failed`, a ticket),
// so that the block goes on or leaves as a whole.
//
// Measured (all generations of theta 0.5, host reads included) against two launches per
// generation, one that classifies and scans and one that reads the frontier again and emits:
// 0.84 -> 0.50 ms (1M clustered particles, leaf 8), 0.51 -> 0.28 ms (200k), 0.24 -> 0.13 ms
// (2000).  GEN_ITEMS 8 (fewer, longer tiles) 0.53 / 0.36 / 0.16 ms, 2: 0.61 / 0.30 / 0.12 ms.
constexpr int GEN_ITEMS = 4;
constexpr int GEN_TILE = TRAV_THREADS * GEN_ITEMS;
constexpr int GEN_FIRST = 16, GEN_BATCH = 8;  // generations before the first / next host read
constexpr int GEN_BLOCKS = 4;  // resident per SM
constexpr unsigned LOOK_LIMIT = 1u << 22;

struct TravState {
    i64 nf[2];          // frontier size of even / odd generations
    i64 n_m2l, n_p2p;   // pairs listed so far
    i64 overflow;       // a list or the next frontier outgrew its buffer
    i64 need_m2l, need_p2p, need_frontier;
    i64 failed;         // a wait ran out
    unsigned ticket[4];  // tiles taken, of generation g at g mod 4
};

// A tile's counts of a generation (its own, or with all tiles before it): m2l and p2p pairs
// in the halves of `lists`, next-frontier pairs in `next`.  `ready` is 2 g + 1 once `own` is
// there and 2 g + 2 once `all` is, g the generation's number from 0.
struct TileCounts {
    unsigned long long lists;
    unsigned long long next;
};
struct TileState {
    TileCounts own, all;
    unsigned ready, pad[3];
};

template <bool DUAL>
__device__ __forceinline__ int classify_pair(const NodeRec* t, const NodeRec* s, double theta,
                                             FPair pr) {
    if (DUAL) return classify_dual(pr.a, pr.b, t, s, theta);
    return classify_mutual(pr.a, pr.b, t, theta);
}

__global__ void k_gen_init(TravState* st, FPair* frontier, TileState* tile, i64 tiles) {
    td3_chain_wait();
    td3_chain_release();
    const i64 i = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < tiles) tile[i].ready = 0;
    if (i) return;
    *st = TravState{};
    st->nf[0] = 1;
    frontier[0] = FPair{0, 0};
}

__device__ __forceinline__ unsigned load_acquire(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void store_release(unsigned* p, unsigned v) {
    asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// The counts of all tiles before `tile` (one warp; every lane returns them): 32 tiles at a
// time, the lanes nearest first, up to the nearest tile whose `all` is there.
__device__ TileCounts look_back(TileState* state, i64 tile, unsigned own_ready, unsigned limit,
                                bool* failed) {
    const int lane = threadIdx.x & 31;
    TileCounts sum{0, 0};
    for (i64 at = tile - 1; at >= 0; at -= 32) {
        const i64 t = at - lane;
        unsigned ready = own_ready + 1;  // before the first tile: nothing, known
        if (t >= 0) {
            ready = 0;
            for (unsigned polls = 0;
                 polls < limit && (ready = load_acquire(&state[t].ready)) < own_ready; ++polls)
                __nanosleep(20);
        }
        if (__any_sync(0xffffffffu, ready < own_ready)) {
            *failed = true;
            return sum;
        }
        const unsigned known = __ballot_sync(0xffffffffu, ready > own_ready);
        const int last = known ? __ffs(known) - 1 : 31;  // the nearest tile with `all`
        TileCounts c{0, 0};
        if (t >= 0 && lane <= last) {
            const TileCounts* from = lane == last && known ? &state[t].all : &state[t].own;
            c.lists = __ldcg(&from->lists);
            c.next = __ldcg(&from->next);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            c.lists += __shfl_xor_sync(0xffffffffu, c.lists, o);
            c.next += __shfl_xor_sync(0xffffffffu, c.next, o);
        }
        sum.lists += c.lists;
        sum.next += c.next;
        if (known) break;
    }
    return sum;
}

// One generation.  A warp takes 32 * GEN_ITEMS consecutive pairs of a tile (round r, lane l:
// pair first + 32 r + l); ballots rank a round's outputs, in frontier order.
template <bool DUAL>
__global__ void __launch_bounds__(TRAV_THREADS, GEN_BLOCKS)
k_generation(const FPair* __restrict__ frontier, TravState* st, int gen, unsigned look_limit,
             const NodeRec* __restrict__ t_rec, const NodeRec* __restrict__ s_rec, double theta,
             TileState* tile_state, Pair* __restrict__ m2l, i64 m2l_capacity,
             Pair* __restrict__ p2p, i64 p2p_capacity, FPair* __restrict__ next,
             i64 frontier_capacity) {
    constexpr int WARPS = TRAV_THREADS / 32;
    __shared__ unsigned warp_m2l[WARPS], warp_p2p[WARPS], warp_next[WARPS];
    __shared__ i64 base_m2l_s, base_p2p_s, base_next_s, nf_s, listed_m2l_s, listed_p2p_s;
    __shared__ unsigned taken;
    td3_chain_wait();
    td3_chain_release();
    const int parity = gen & 1, lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const unsigned before = (1u << lane) - 1u;
    // read before this block takes a tile: the last tile's block moves them on (a generation
    // after a failed one, whose frontier has holes, is empty)
    if (threadIdx.x == 0) {
        const i64 size = st->nf[parity], m = st->n_m2l, p = st->n_p2p, stop = st->failed;
        nf_s = stop ? 0 : size;
        listed_m2l_s = m;
        listed_p2p_s = p;
    }
    __syncthreads();
    const i64 nf = nf_s, listed_m2l = listed_m2l_s, listed_p2p = listed_p2p_s;
    const i64 tiles = (nf + GEN_TILE - 1) / GEN_TILE;
    const unsigned own_ready = 2u * (unsigned)gen + 1u;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        st->ticket[(gen + 2) & 3] = 0;
        if (tiles == 0) st->nf[parity ^ 1] = 0;
    }
    if ((i64)blockIdx.x >= tiles) return;  // the others take every tile
    for (;;) {
        if (threadIdx.x == 0) taken = atomicAdd(&st->ticket[gen & 3], 1u);
        __syncthreads();
        const i64 tile = taken;
        if (tile >= tiles) return;
        const i64 first = tile * GEN_TILE + (i64)wib * 32 * GEN_ITEMS;
        FPair pr[GEN_ITEMS];
        int act[GEN_ITEMS];
        unsigned n_m2l = 0, n_p2p = 0, n_next = 0;  // the warp's
#pragma unroll
        for (int r = 0; r < GEN_ITEMS; ++r) {
            const i64 k = first + r * 32 + lane;
            pr[r] = k < nf ? frontier[k] : FPair{0, 0};
        }
#pragma unroll
        for (int r = 0; r < GEN_ITEMS; ++r) {
            const i64 k = first + r * 32 + lane;
            act[r] = k < nf ? classify_pair<DUAL>(t_rec, s_rec, theta, pr[r]) : ACT_NONE;
        }
#pragma unroll
        for (int r = 0; r < GEN_ITEMS; ++r) {
            n_m2l += __popc(__ballot_sync(0xffffffffu, act[r] == ACT_M2L));
            n_p2p += __popc(__ballot_sync(0xffffffffu, act[r] == ACT_P2P));
            n_next += 4 * __popc(__ballot_sync(0xffffffffu, act[r] >= ACT_SPLIT_A));
            if (!DUAL) n_next += 10 * __popc(__ballot_sync(0xffffffffu, act[r] == ACT_SELF));
        }
        if (lane == 0) {
            warp_m2l[wib] = n_m2l;
            warp_p2p[wib] = n_p2p;
            warp_next[wib] = n_next;
        }
        __syncthreads();
        if (wib == 0) {
            // the tile's counts, published; then the tiles' before it
            TileCounts own{0, 0};
            for (int w = 0; w < WARPS; ++w) {
                own.lists += warp_m2l[w] | ((unsigned long long)warp_p2p[w] << 32);
                own.next += warp_next[w];
            }
            TileState* mine = tile_state + tile;
            if (lane == 0 && tile) {
                __stcg(&mine->own.lists, own.lists);
                __stcg(&mine->own.next, own.next);
                store_release(&mine->ready, own_ready);
            }
            bool failed = false;
            const TileCounts pre = look_back(tile_state, tile, own_ready, look_limit, &failed);
            if (lane == 0) {
                const TileCounts all{pre.lists + own.lists, pre.next + own.next};
                if (failed) {
                    st->failed = 1;
                    st->nf[parity ^ 1] = 0;
                    taken = 0xffffffffu;
                } else {
                    __stcg(&mine->all.lists, all.lists);
                    __stcg(&mine->all.next, all.next);
                    store_release(&mine->ready, own_ready + 1);
                    base_m2l_s = listed_m2l + (i64)(pre.lists & 0xffffffffull);
                    base_p2p_s = listed_p2p + (i64)(pre.lists >> 32);
                    base_next_s = (i64)pre.next;
                    if (tile == tiles - 1) {
                        const i64 total_m2l = listed_m2l + (i64)(all.lists & 0xffffffffull);
                        const i64 total_p2p = listed_p2p + (i64)(all.lists >> 32);
                        const i64 nn = (i64)all.next;
                        if (total_m2l > m2l_capacity || total_p2p > p2p_capacity ||
                            nn > frontier_capacity) {
                            st->overflow = 1;
                            st->need_m2l = total_m2l;
                            st->need_p2p = total_p2p;
                            st->need_frontier = nn;
                            st->nf[parity ^ 1] = 0;
                        } else {
                            st->n_m2l = total_m2l;
                            st->n_p2p = total_p2p;
                            st->nf[parity ^ 1] = nn;
                        }
                    }
                }
            }
        }
        __syncthreads();
        if (taken == 0xffffffffu) return;
        i64 at_m2l = base_m2l_s, at_p2p = base_p2p_s, at_next = base_next_s;
        for (int w = 0; w < wib; ++w) {
            at_m2l += warp_m2l[w];
            at_p2p += warp_p2p[w];
            at_next += warp_next[w];
        }
#pragma unroll
        for (int r = 0; r < GEN_ITEMS; ++r) {
            const unsigned bm = __ballot_sync(0xffffffffu, act[r] == ACT_M2L);
            const unsigned bp = __ballot_sync(0xffffffffu, act[r] == ACT_P2P);
            const unsigned bs = __ballot_sync(0xffffffffu, act[r] >= ACT_SPLIT_A);
            const unsigned bb = DUAL ? 0u : __ballot_sync(0xffffffffu, act[r] == ACT_SELF);
            const i64 to = at_next + 4 * __popc(bs & before) + 10 * __popc(bb & before);
            // outputs past a buffer's end are left out: the last tile reports the overflow
            switch (act[r]) {
                case ACT_NONE: break;
                case ACT_M2L: {
                    const i64 j = at_m2l + __popc(bm & before);
                    if (j < m2l_capacity) m2l[j] = Pair{pr[r].a, pr[r].b};
                    break;
                }
                case ACT_P2P: {
                    const i64 j = at_p2p + __popc(bp & before);
                    if (j < p2p_capacity) p2p[j] = Pair{pr[r].a, pr[r].b};
                    break;
                }
                case ACT_SELF: {
                    if (to + 10 > frontier_capacity) break;
                    const int f = t_rec[pr[r].a].child;
                    i64 j = to;
                    for (int c1 = 0; c1 < 4; ++c1)
                        for (int d = c1; d < 4; ++d) next[j++] = FPair{f + c1, f + d};
                    break;
                }
                case ACT_SPLIT_A: {
                    if (to + 4 > frontier_capacity) break;
                    const int f = t_rec[pr[r].a].child;
                    for (int c1 = 0; c1 < 4; ++c1) next[to + c1] = FPair{f + c1, pr[r].b};
                    break;
                }
                default: {
                    if (to + 4 > frontier_capacity) break;
                    const int f = (DUAL ? s_rec : t_rec)[pr[r].b].child;
                    for (int c1 = 0; c1 < 4; ++c1) next[to + c1] = FPair{pr[r].a, f + c1};
                    break;
                }
            }
            at_m2l += __popc(bm);
            at_p2p += __popc(bp);
            at_next += 4 * __popc(bs) + 10 * __popc(bb);
        }
        __syncthreads();  // the tile's counts and slots have been read
    }
}

struct TraverseBuffers {
    FPair* frontier[2];
    TileState* tile;
    TravState* state;
    NodeRec* rec[2];  // target (and source) tree records
};

i64 gen_tiles(i64 frontier_cap) { return (frontier_cap + GEN_TILE - 1) / GEN_TILE; }

size_t traverse_workspace(i64 frontier_cap, i64 n_records) {
    return 2 * td3_ws_bytes<FPair>(frontier_cap) +
           td3_ws_bytes<TileState>(gen_tiles(frontier_cap)) + td3_ws_bytes<TravState>(1) +
           td3_ws_bytes<NodeRec>(n_records) + 512;
}

bool take_traverse(Workspace& w, i64 frontier_cap, i64 n_t, i64 n_s, TraverseBuffers& b) {
    b.frontier[0] = w.take<FPair>(frontier_cap);
    b.frontier[1] = w.take<FPair>(frontier_cap);
    b.tile = w.take<TileState>(gen_tiles(frontier_cap));
    b.state = w.take<TravState>(1);
    b.rec[0] = w.take<NodeRec>(n_t);
    b.rec[1] = n_s ? w.take<NodeRec>(n_s) : b.rec[0];
    return b.rec[1] != nullptr;
}

int launch_records(i64 count, const double* center, const double* half, const i64* start,
                    const i64* end, const i64* child, NodeRec* rec, cudaStream_t stream) {
    TD3_TRY(td3_launch_chained(k_node_records, td3_blocks(count, 256), 256, 0, stream, count,
                               center, half, start, end, child, rec));
    return TD3_OK;
}

// The generations from (root, root) until the frontier is empty; sizes as the entry
// points document them.
template <bool DUAL>
int run_generations(const NodeRec* t, const NodeRec* s, double theta, Pair* m2l,
                    i64 m2l_capacity, Pair* p2p, i64 p2p_capacity, i64 frontier_capacity,
                    int64_t* sizes, const TraverseBuffers& b, unsigned look_limit,
                    cudaStream_t stream) {
    i64 tiles = gen_tiles(frontier_capacity);
    unsigned grid = (unsigned)(tiles < 148 * 4 ? tiles : 148 * 4);
    TD3_TRY(td3_launch_chained(k_gen_init, td3_blocks(tiles, 256), 256, 0, stream, b.state,
                               b.frontier[0], b.tile, tiles));
    TD3_CHECK_LAUNCH();
    sizes[0] = sizes[1] = sizes[2] = sizes[3] = 0;
    for (int gen = 0;;) {
        for (const int stop = gen + (gen ? GEN_BATCH : GEN_FIRST); gen < stop; ++gen) {
            const int parity = gen & 1;
            TD3_TRY(td3_launch_chained(k_generation<DUAL>, grid, TRAV_THREADS, 0, stream,
                                       (const FPair*)b.frontier[parity], b.state, gen, look_limit,
                                       t, s, theta, b.tile, m2l, m2l_capacity, p2p, p2p_capacity,
                                       b.frontier[parity ^ 1], frontier_capacity));
        }
        TD3_CHECK_LAUNCH();
        TravState h;
        TD3_TRY(cudaMemcpyAsync(&h, b.state, sizeof(h), cudaMemcpyDeviceToHost, stream));
        TD3_TRY(cudaStreamSynchronize(stream));
        if (h.failed) {
            td3_set_error("a generation of the traversal did not complete (a bounded wait ran out)");
            return TD3_ECUDA;
        }
        if (h.overflow) {
            sizes[0] = h.need_m2l;
            sizes[1] = h.need_p2p;
            sizes[2] = h.need_frontier;
            sizes[3] = -1;
            return TD3_ENEEDMORE;
        }
        if (h.nf[gen & 1] == 0) {
            sizes[0] = h.n_m2l;
            sizes[1] = h.n_p2p;
            return TD3_OK;
        }
    }
}

// ------------------------------------------------------------------ pair CSR
__global__ void k_csr_keys(const Pair* __restrict__ pairs, i64 count, int mutual, unsigned invalid,
                           unsigned* __restrict__ keys, unsigned* __restrict__ vals) {
    td3_chain_wait();
    td3_chain_release();
    i64 p = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= count) return;
    Pair pr = pairs[p];
    if (mutual) {
        keys[2 * p] = (unsigned)pr.a;
        vals[2 * p] = (unsigned)pr.b;
        if (pr.a != pr.b) {
            keys[2 * p + 1] = (unsigned)pr.b;
            vals[2 * p + 1] = (unsigned)pr.a;
        } else {
            keys[2 * p + 1] = invalid;
            vals[2 * p + 1] = 0;
        }
    } else {
        keys[p] = (unsigned)pr.a;
        vals[p] = (unsigned)pr.b;
    }
}

// The CSR from the sorted entries, one thread per position j in [0, e]: partners (int64)
// and, when asked, the row of every entry (int32); and row_start[d] = the first sorted
// position with key >= d (keys sorted, the invalid key n_nodes last), position j setting
// the rows between its predecessor's key and its own.
__global__ void k_csr_out(const unsigned* __restrict__ vals, const unsigned* __restrict__ keys,
                          i64 e, i64 n_nodes, i64* __restrict__ row_start,
                          i64* __restrict__ partners, int* __restrict__ entry_row) {
    td3_chain_wait();
    td3_chain_release();
    i64 j = (i64)blockIdx.x * blockDim.x + threadIdx.x;
    if (j > e) return;
    i64 prev = j == 0 ? -1 : (i64)keys[j - 1];
    i64 cur = n_nodes;
    if (j < e) {
        unsigned key = keys[j];
        partners[j] = vals[j];
        if (entry_row) entry_row[j] = (int)key;
        cur = (i64)key < n_nodes ? (i64)key : n_nodes;
    }
    for (i64 d = prev + 1; d <= cur; ++d) row_start[d] = j;
}

int bits_for(i64 v) {
    int b = 1;
    while (b < 32 && ((i64)1 << b) <= v) ++b;
    return b;
}

}  // namespace

extern "C" size_t td3_fmm_traverse_workspace_size(int64_t frontier_capacity, int64_t n_nodes) {
    return traverse_workspace(frontier_capacity, n_nodes);
}

extern "C" int td3_fmm_traverse_polls(const double* node_center, const double* node_half,
                                      const int64_t* node_start, const int64_t* node_end,
                                      const int64_t* node_child, int64_t n_nodes, double theta,
                                      int64_t* m2l, int64_t m2l_capacity, int64_t* p2p,
                                      int64_t p2p_capacity, int64_t frontier_capacity,
                                      int64_t* sizes, int64_t polls, void* workspace,
                                      size_t workspace_bytes, void* stream) {
    if (frontier_capacity < 1 || m2l_capacity < 0 || p2p_capacity < 0) return TD3_EINVAL;
    if (n_nodes < 1 || n_nodes > 0x7fffffffLL || polls < 0 || polls > LOOK_LIMIT) return TD3_EINVAL;
    Workspace w(workspace, workspace_bytes);
    TraverseBuffers b;
    if (!take_traverse(w, frontier_capacity, n_nodes, 0, b)) return TD3_EWORKSPACE;
    cudaStream_t s = td3_stream(stream);
    TD3_TRY_RC(launch_records(n_nodes, node_center, node_half, node_start, node_end, node_child,
                              b.rec[0], s));
    return run_generations<false>(b.rec[0], b.rec[0], theta, reinterpret_cast<Pair*>(m2l),
                                  m2l_capacity, reinterpret_cast<Pair*>(p2p), p2p_capacity,
                                  frontier_capacity, sizes, b, (unsigned)polls, s);
}

extern "C" int td3_fmm_traverse(const double* node_center, const double* node_half,
                                const int64_t* node_start, const int64_t* node_end,
                                const int64_t* node_child, int64_t n_nodes, double theta,
                                int64_t* m2l, int64_t m2l_capacity, int64_t* p2p,
                                int64_t p2p_capacity, int64_t frontier_capacity, int64_t* sizes,
                                void* workspace, size_t workspace_bytes, void* stream) {
    return td3_fmm_traverse_polls(node_center, node_half, node_start, node_end, node_child, n_nodes,
                                  theta, m2l, m2l_capacity, p2p, p2p_capacity, frontier_capacity,
                                  sizes, LOOK_LIMIT, workspace, workspace_bytes, stream);
}

extern "C" int td3_dual_traverse(const double* t_center, const double* t_half,
                                 const int64_t* t_start, const int64_t* t_end,
                                 const int64_t* t_child, int64_t t_nodes, const double* s_center,
                                 const double* s_half, const int64_t* s_start,
                                 const int64_t* s_end, const int64_t* s_child, int64_t s_nodes,
                                 double theta, int64_t* m2l, int64_t m2l_capacity, int64_t* p2p,
                                 int64_t p2p_capacity, int64_t frontier_capacity, int64_t* sizes,
                                 void* workspace, size_t workspace_bytes, void* stream) {
    if (frontier_capacity < 1 || m2l_capacity < 0 || p2p_capacity < 0) return TD3_EINVAL;
    if (t_nodes < 1 || s_nodes < 1 || t_nodes > 0x7fffffffLL || s_nodes > 0x7fffffffLL)
        return TD3_EINVAL;
    Workspace w(workspace, workspace_bytes);
    TraverseBuffers b;
    if (!take_traverse(w, frontier_capacity, t_nodes, s_nodes, b)) return TD3_EWORKSPACE;
    cudaStream_t s = td3_stream(stream);
    TD3_TRY_RC(launch_records(t_nodes, t_center, t_half, t_start, t_end, t_child, b.rec[0], s));
    TD3_TRY_RC(launch_records(s_nodes, s_center, s_half, s_start, s_end, s_child, b.rec[1], s));
    return run_generations<true>(b.rec[0], b.rec[1], theta, reinterpret_cast<Pair*>(m2l),
                                 m2l_capacity, reinterpret_cast<Pair*>(p2p), p2p_capacity,
                                 frontier_capacity, sizes, b, LOOK_LIMIT, s);
}

extern "C" size_t td3_pair_csr_workspace_size(int64_t count, int mutual, int64_t n_nodes) {
    i64 e = mutual ? 2 * count : count;
    size_t sort = td3_sort_workspace(e), scan = td3_scan_workspace(n_nodes + 1);
    return 4 * td3_ws_bytes<unsigned>(e) + (sort > scan ? sort : scan);
}

extern "C" int td3_pair_csr(const int64_t* pairs, int64_t count, int mutual, int64_t n_nodes,
                            int64_t* row_start, int64_t* partners, int32_t* entry_row,
                            void* workspace, size_t workspace_bytes, void* stream) {
    if (count < 0 || n_nodes < 1 || n_nodes >= 0x7fffffffLL) return TD3_EINVAL;
    cudaStream_t s = td3_stream(stream);
    if (count == 0) {
        TD3_TRY(cudaMemsetAsync(row_start, 0, sizeof(i64) * (n_nodes + 1), s));
        return TD3_OK;
    }
    i64 e = mutual ? 2 * count : count;
    Workspace w(workspace, workspace_bytes);
    unsigned* k0 = w.take<unsigned>(e);
    unsigned* k1 = w.take<unsigned>(e);
    unsigned* v0 = w.take<unsigned>(e);
    unsigned* v1 = w.take<unsigned>(e);
    if (!v1) return TD3_EWORKSPACE;
    TD3_TRY(td3_launch_chained(k_csr_keys, td3_blocks(count, 256), 256, 0, s,
                               reinterpret_cast<const Pair*>(pairs), count, mutual,
                               (unsigned)n_nodes, k0, v0));
    TD3_CHECK_LAUNCH();
    unsigned *ko, *vo;
    TD3_TRY_RC(td3_radix_sort_u32(k0, k1, v0, v1, e, bits_for(n_nodes), &ko, &vo, w.base + w.used,
                                  w.size - w.used, s));
    // the row offsets from the boundaries between equal keys of the sorted entries; valid
    // entries sort before the invalid key n_nodes (row_start[n_nodes] of them), the entries
    // after them are widened too (partners holds e slots), so no host read
    TD3_TRY(td3_launch_chained(k_csr_out, td3_blocks(e + 1, 256), 256, 0, s, vo, ko, e, n_nodes,
                               row_start, partners, entry_row));
    TD3_CHECK_LAUNCH();
    return TD3_OK;
}
