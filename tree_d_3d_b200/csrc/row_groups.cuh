// The walk of a warp over CSR rows of an M2L with a lane per entry (cart_m2l.cuh,
// m2l_log_rows.cu): groups of ROW_GL lanes take the warp's rows in order, lane i of a group
// the entries i, i + ROW_GL, ... of its row; rows above LONG_ROW entries are taken by the
// whole warp first.  Each row is summed by one group or warp in a fixed order.
//
// Small trees (FEW_ROWS): a group needs 9 rounds for a row of 35 entries however few rows
// there are, the whole warp 2 per row; the log M2L of 5000 particles at p = 12 took 0.079 ms
// with groups against 0.060 ms for the form before, 0.034 ms with whole warps.
//
// Groups of 4: a row of 35 entries, the mean of the FMM's lists at theta 0.5, fills 97 % of
// its lanes' rounds (87 % with groups of 8).
#pragma once

#include "common.cuh"

constexpr int ROW_GL = 4;                // lanes per row
constexpr int ROW_GROUPS = 32 / ROW_GL;  // rows in flight per warp
constexpr unsigned ROW_LEADERS = 0xffffffffu / ((1u << ROW_GL) - 1u);  // each group's lane 0
static_assert(ROW_GL == 4 && ROW_LEADERS == 0x11111111u, "the row sums add four lanes by name");
constexpr int LONG_ROW = 256;            // rows longer than this are taken by the whole warp,
constexpr int FEW_ROWS = 6;              // or, with at most so many rows per warp,
constexpr int LONG_OF_FEW = 8;           // rows longer than this
constexpr int ROW_COST = 8;              // entries a row counts for in the warps' shares
constexpr unsigned FULL_WARP = 0xffffffffu;

// Warp `warp` of `warps` takes a run of whole rows with an even share of the cost, entries +
// ROW_COST per row.  For every round of entries:
//   fetch(src, row)             all lanes: starts the loads for the lanes' sources (-1: none);
//   ready(to_src)               all lanes: the copies are done (to_src: the next round's);
//   translate()                 the lanes with an entry;
//   finish(row, whole, mask)    the lanes (mask) whose row has had its last entry: adds the
//                               row's sums to the locals and clears them (whole: every lane of
//                               the warp holds a part of the row's).
template <class Fetch, class Ready, class Translate, class Finish>
__device__ __forceinline__ void walk_rows(const i64* __restrict__ row_start,
                                          const i64* __restrict__ partners, i64 n_rows, i64 warp,
                                          i64 warps, Fetch fetch, Ready ready,
                                          Translate translate, Finish finish) {
    const int lane = threadIdx.x & 31, g = lane / ROW_GL, gl = lane % ROW_GL;
    const i64 total = row_start[n_rows] + ROW_COST * n_rows, share = (total + warps - 1) / warps;
    auto first_row_at = [&](i64 c) {
        i64 lo = 0, hi = n_rows;
        while (lo < hi) {
            const i64 mid = (lo + hi) >> 1;
            if (row_start[mid] + ROW_COST * mid < c) lo = mid + 1;
            else hi = mid;
        }
        return lo;
    };
    const i64 da = first_row_at(warp * share);
    const i64 db = warp + 1 == warps ? n_rows : first_row_at((warp + 1) * share);
    if (da >= db) return;
    const int long_row = n_rows <= FEW_ROWS * warps ? LONG_OF_FEW : LONG_ROW;
    i64 scan = da;       // long rows are looked for from `scan` on, 32 rows at a time
    unsigned longs = 0;  // those found in the 32 rows before `scan`
    auto next_long = [&]() -> i64 {
        while (!longs && scan < db) {
            const i64 r = scan + lane;
            longs = __ballot_sync(FULL_WARP, r < db && row_start[r + 1] - row_start[r] > long_row);
            scan += 32;
        }
        if (!longs) return -1;
        const int k = __ffs(longs) - 1;
        longs &= longs - 1;
        return scan - 32 + k;
    };
    // A lane's place: row da + d (d < 0: none), entries e0 + cur, ... of it left (32-bit
    // distances from the warp's first row and entry).
    const i64 e0 = row_start[da];
    struct Place {
        int d, cur, end;
        bool filled;  // the row has entries to sum here
    };
    auto claim = [&](i64 row, bool whole) {
        Place at{row < db ? (int)(row - da) : -1, 0, 0, false};
        if (at.d < 0) return at;
        const int start = (int)(row_start[row] - e0);
        at.cur = start + (whole ? lane : gl);
        at.end = (int)(row_start[row + 1] - e0);
        if (!whole && at.end - start > long_row) at.end = start;  // done as a long row
        at.filled = at.end > start;
        return at;
    };
    auto partner = [&](const Place& at) {
        return at.d >= 0 && at.cur < at.end ? (int)partners[e0 + at.cur] : -1;
    };
    i64 next = da + ROW_GROUPS;  // the first row that no group has taken
    i64 row = next_long();
    bool whole = row >= 0;
    Place at = whole ? claim(row, true) : claim(da + g, false);
    int src = partner(at);
    while (__any_sync(FULL_WARP, at.d >= 0)) {
        const bool work = __any_sync(FULL_WARP, src >= 0);
        if (work) fetch(src, da + at.d);
        // while the copies are under way: where each lane goes next, and its partner there
        const bool was_whole = whole;
        Place to = at;
        to.cur += whole ? 32 : ROW_GL;
        // lane 0 of a group (of the warp) has the last entries: its row is done with it
        const int lead = __shfl_sync(FULL_WARP, to.cur, whole ? 0 : lane & ~(ROW_GL - 1));
        const bool done = at.d >= 0 && lead >= at.end;
        const unsigned dm = __ballot_sync(FULL_WARP, done);
        const unsigned sums = __ballot_sync(FULL_WARP, done && at.filled);
        if (dm) {
            if (whole) {
                row = next_long();
                whole = row >= 0;
                to = whole ? claim(row, true) : claim(da + g, false);
            } else {
                // the finished groups take the next rows, in group order
                const unsigned gm = dm & ROW_LEADERS;
                if (done) to = claim(next + __popc(gm & ((1u << (ROW_GL * g)) - 1u)), false);
                next += __popc(gm);
            }
        }
        const int to_src = partner(to);
        if (work) {
            ready(to_src);
            if (src >= 0) translate();
        }
        if (done && at.filled) finish(da + at.d, was_whole, sums);
        __syncwarp();
        at = to;
        src = to_src;
    }
}

__device__ __forceinline__ unsigned shared_address(const void* p) {
    return (unsigned)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void copies_done() {
    asm volatile("cp.async.wait_all;" ::: "memory");
}
