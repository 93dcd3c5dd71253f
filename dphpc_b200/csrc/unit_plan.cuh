// Building the unit lists of the row-segment kernels (once per upload, all on the device).
//
// A list is made from ENTRIES, each a run of consecutive nonzeros of one row (a whole row; the part of a row inside a
// column panel; the leader of a row group; nothing).  Two kernels: the first sums the units of every tile of entries, the
// second scans inside its tile, adds the sums of the tiles before it, and writes headers and column indices with one
// thread per slot -- balanced whatever the run lengths, and nothing but the list itself goes to memory.
#pragma once

#include "device_utils.cuh"
#include "kernel_rowseg.cuh"
#include "plan_kernels.cuh"

namespace sddmm {

// ---- entries -> runs.  (A row_ptr that has not been validated yet may be anything: runs outside [0, nnz) are empty.) ----
// settled(pc): the runs themselves, where the row statistics have a say (RunsOfForms); wanted(): whether k_unit_build is to list them;
// sorted(): whether they need sorted columns; ordered(): whether a list that may be ordered by size is
struct RunsOfRows {   // one entry per row: the whole row
    static constexpr bool kChosen = false;
    __device__ __forceinline__ const RunsOfRows &settled(const PlanCounters *) const { return *this; }
    __device__ __forceinline__ bool wanted(const PlanCounters *) const { return true; }
    __device__ __forceinline__ bool sorted() const { return false; }
    __device__ __forceinline__ bool ordered() const { return true; }
    const int32_t *rp;
    const int32_t *col;
    int32_t M, nnz;
    __device__ __forceinline__ int32_t row(int64_t q) const { return static_cast<int32_t>(q); }
    __device__ __forceinline__ void run(int64_t q, int32_t &s, int32_t &e) const {
        s = rp[q];
        e = rp[q + 1];
        if (s < 0 || e < s || e > nnz) s = e = 0;
    }
};
// One entry per (panel, row), panel-major.  Needs non-decreasing column indices inside a row.
// long_rows > 0: only rows of at least that many nonzeros are cut into column panels (panels 0 .. panels-2, panel_cols
// columns each); the shorter rows follow whole, as the last "panel" of the list -- a run of one or two nonzeros would
// leave most of a segment's slots empty.
struct RunsOfPanels {
    static constexpr bool kChosen = false;
    const int32_t *rp;
    const int32_t *col;
    int32_t M, nnz, panels, panel_cols, long_rows;
    bool by_size = true;
    const int32_t *cuts = nullptr;   // where panel p + 1 starts in row i, at p * M + i (k_panel_cuts; null: it is looked for, in each kernel)
    __device__ __forceinline__ const RunsOfPanels &settled(const PlanCounters *) const { return *this; }
    __device__ __forceinline__ bool wanted(const PlanCounters *) const { return true; }
    __device__ __forceinline__ bool sorted() const { return panels > 1; }
    __device__ __forceinline__ bool ordered() const { return by_size; }
    __device__ __forceinline__ int32_t real_panels() const { return long_rows > 0 ? panels - 1 : panels; }   // (without the short rows)
    __device__ __forceinline__ void split(int64_t q, int32_t &p, int32_t &i) const {   // (a 64-bit division is several times a 32-bit one)
        if (panels == 1) {
            p = 0;
            i = static_cast<int32_t>(q);
        } else if ((q >> 32) == 0) {
            p = static_cast<int32_t>(static_cast<uint32_t>(q) / static_cast<uint32_t>(M));
            i = static_cast<int32_t>(static_cast<uint32_t>(q) - static_cast<uint32_t>(p) * static_cast<uint32_t>(M));
        } else {
            p = static_cast<int32_t>(q / M);
            i = static_cast<int32_t>(q - static_cast<int64_t>(p) * M);
        }
    }
    __device__ __forceinline__ int32_t row(int64_t q) const {
        int32_t p, i;
        split(q, p, i);
        return i;
    }
    __device__ __forceinline__ bool bounds(int32_t i, int32_t &a, int32_t &b) const {
        a = rp[i];
        b = rp[i + 1];
        return a >= 0 && b >= a && b <= nnz;
    }
    __device__ __forceinline__ void run(int64_t q, int32_t &s, int32_t &e) const {
        int32_t p, i, a, b;
        split(q, p, i);
        s = e = 0;
        if (!bounds(i, a, b)) return;
        if (long_rows > 0) {
            const bool is_long = b - a >= long_rows;
            if (p == panels - 1) {           // the short rows, whole
                s = a;
                e = is_long ? a : b;
                return;
            }
            if (!is_long) return;
        }
        auto start = [&](int32_t k) -> int32_t {
            return cuts ? cuts[static_cast<int64_t>(k - 1) * M + i] : lower_col(col, a, b, static_cast<int64_t>(k) * panel_cols);
        };
        s = p == 0 ? a : start(p);
        e = p == real_panels() - 1 ? b : start(p + 1);
        if (e < s) e = s;                    // (unsorted columns: the list will not be used)
    }
};
// The forms that a list over the whole matrix may take, and which one the row statistics choose: on the device for a list that is
// enqueued before the host has seen them, on the host to know which one that was.
struct ListForms {
    int32_t plain = 1, plain_cols = 0;   // column panels for every row (1: whole rows)
    int32_t longs = 1, long_cols = 0;    // panels for the rows of at least long_rows nonzeros, the others being one more
    int32_t long_rows = 0;               // (0: no such form)
    bool long_always = false;            // whatever those rows hold
    bool plain_for_8 = false;            // plain panels only where most rows have 8 nonzeros or more
    bool plain_by_size = false, long_by_size = false;
    struct Choice {
        int32_t panels, panel_cols, long_rows;
        bool by_size;
    };
    // what the choice rests on, of the rows of one length bin (hist, hist_nnz: bin 0 holds the empty rows)
    struct Rows {
        unsigned long long rows = 0, of_8 = 0, in_long = 0;
    };
    __host__ __device__ __forceinline__ Rows of_bin(const PlanCounters *pc, int b) const {
        Rows r;
        if (b < 1 || b >= SDDMM_B200_HIST_BINS) return r;
        r.rows = pc->hist[b];
        r.of_8 = b >= 4 ? r.rows : 0;
        r.in_long = (1ll << (b - 1)) >= long_rows ? pc->hist_nnz[b] : 0;
        return r;
    }
    __host__ __device__ __forceinline__ Choice of_rows(const Rows &r, int64_t nnz) const {
        // panels for the long rows only pay when those hold a good share of the nonzeros, 40 %
        const bool mostly_long = 5 * r.in_long >= 2 * static_cast<unsigned long long>(nnz);
        if (long_rows > 0 && (long_always || mostly_long)) return Choice{longs + 1, long_cols, long_rows, long_by_size};
        // a mean that barely pays for panels has to be that of most rows, not of a few long ones: 60 % of them of 8 nonzeros or more
        if (plain > 1 && plain_for_8 && 10 * r.of_8 < 6 * r.rows) return Choice{1, plain_cols, 0, plain_by_size};
        return Choice{plain, plain_cols, 0, plain_by_size};
    }
    Choice choose(const PlanCounters *pc, int64_t nnz) const {
        Rows r;
        for (int b = 1; b < SDDMM_B200_HIST_BINS; ++b) {
            const Rows bin = of_bin(pc, b);
            r.rows += bin.rows;
            r.of_8 += bin.of_8;
            r.in_long += bin.in_long;
        }
        return of_rows(r, nnz);
    }
    // (a bin per lane, by whole warps: bin after bin, the loads one after the other, every block of a list takes 4 us longer)
    __device__ __forceinline__ Choice choose_by_warp(const PlanCounters *pc, int64_t nnz) const {
        static_assert(SDDMM_B200_HIST_BINS <= 32, "a length bin per lane");
        Rows r = of_bin(pc, static_cast<int>(threadIdx.x & 31));
        for (int o = 16; o > 0; o >>= 1) {
            r.rows += __shfl_xor_sync(kFullMask, r.rows, o);
            r.of_8 += __shfl_xor_sync(kFullMask, r.of_8, o);
            r.in_long += __shfl_xor_sync(kFullMask, r.in_long, o);
        }
        return of_rows(r, nnz);
    }
};
struct RunsOfForms {
    static constexpr bool kChosen = true;
    const int32_t *rp;
    const int32_t *col;
    int32_t M, nnz;
    ListForms forms;
    int32_t *cuts;       // room for this many starts of panels
    int64_t cuts_room;
    bool have_sums;      // of whole rows
    bool whole_apart;    // whole rows are listed by a kernel of their own (WholeRowsOfForms)
    __device__ __forceinline__ bool wanted(const PlanCounters *pc) const { return !whole_apart || forms.choose_by_warp(pc, nnz).panels > 1; }
    __device__ __forceinline__ RunsOfPanels settled(const PlanCounters *pc) const {   // (by whole warps)
        const ListForms::Choice c = forms.choose_by_warp(pc, nnz);
        RunsOfPanels r{rp, col, M, nnz, c.panels, c.panel_cols, c.long_rows, c.by_size};
        if (static_cast<int64_t>(r.real_panels() - 1) * M <= cuts_room) r.cuts = cuts;
        return r;
    }
};
// ... the whole rows, where these are chosen.  (The kernel for either form takes 111 us for 18 M nonzeros in whole rows, this one 77.)
struct WholeRowsOfForms {
    static constexpr bool kChosen = false;
    RunsOfRows rows;
    ListForms forms;
    __device__ __forceinline__ const RunsOfRows &settled(const PlanCounters *) const { return rows; }
    __device__ __forceinline__ bool wanted(const PlanCounters *pc) const { return forms.choose_by_warp(pc, rows.nnz).panels == 1; }
};
// What may show that a list enqueued before the host has seen the counters will not be used (default: nothing).  Its kernels read
// here only what kernels BEFORE it in its stream have finished: threads of one block that saw a count grow would disagree.
struct ListGate {
    unsigned long long tile_hint = ~0ull;   // nonzeros that look like 64-wide tiles from which on these will be looked for, and found
    double groups_from = -1.0;              // gathers saved by row groups from which on these will be taken (< 0: not looked at)
    int every = 1;                          // of how many groups one is in the sample
    bool columns_scanned = true;            // false: the column scan runs beside (nothing that it counts is read)
};
// Gathers that the best grouping saves, by the sample, and its slot
__host__ __device__ __forceinline__ double group_saving(const unsigned long long *cover, int every, int *slot) {
    double best = 0.0;
    for (int y = 0; y < 9; ++y) {
        const int G = y < 2 ? 2 : y < 5 ? 3 : 4;
        const double saved = static_cast<double>(cover[y]) * every * (1.0 - 1.0 / G);
        if (saved > best) { best = saved; *slot = y; }
    }
    return best;
}
constexpr int kGroupRowMax = 8192;   // (nonzeros of a row) matrices with longer ones are not grouped
__device__ __forceinline__ bool list_unused(const ListGate &gate, const PlanCounters *pc) {
    if (gate.columns_scanned && pc->window_hint >= gate.tile_hint) return true;
    int slot;
    return gate.groups_from >= 0.0 && pc->max_row_nnz <= kGroupRowMax && group_saving(pc->group_cover, gate.every, &slot) >= gate.groups_from;
}

// The starts of the panels, a thread per row: every entry of the list needs two, in both of its kernels, and each is a chain of loads.
// (Whole rows: nothing to do here, nor in k_unit_sums where k_row_stats has left the sums.)
__global__ void __launch_bounds__(kUnitBlock) k_panel_cuts(RunsOfForms given, PlanCounters *__restrict__ pc, ListGate gate) {
    if (list_unused(gate, pc)) return;
    const RunsOfPanels runs = given.settled(pc);
    if (blockIdx.x == 0 && threadIdx.x == 0 && !(given.have_sums && runs.panels == 1)) pc->units = 0;
    if (!runs.cuts || runs.panels == 1) return;
    for (int64_t i = blockIdx.x * static_cast<int64_t>(kUnitBlock) + threadIdx.x; i < runs.M; i += static_cast<int64_t>(gridDim.x) * kUnitBlock) {
        int32_t a, b;
        if (!runs.bounds(static_cast<int32_t>(i), a, b) || b - a < runs.long_rows) continue;   // (not read either)
        for (int32_t k = 1; k < runs.real_panels(); ++k) {
            a = lower_col(runs.col, a, b, static_cast<int64_t>(k) * runs.panel_cols);
            given.cuts[static_cast<int64_t>(k - 1) * runs.M + i] = a;
        }
    }
}
// rows of group g when groups of G rows start at row `first` (group 0 = the rows before it)
__device__ __forceinline__ void unit_group_rows(int32_t g, int32_t G, int32_t first, int32_t M, int32_t &r0, int32_t &r1) {
    r0 = g == 0 ? 0 : first + (g - 1) * G;
    r1 = g == 0 ? first : min(r0 + G, M);
}
struct RunsOfGroups {   // one entry per row: the leader of a matching group speaks for its whole group
    static constexpr bool kChosen = false;
    __device__ __forceinline__ const RunsOfGroups &settled(const PlanCounters *) const { return *this; }
    __device__ __forceinline__ bool wanted(const PlanCounters *) const { return true; }
    __device__ __forceinline__ bool sorted() const { return false; }
    __device__ __forceinline__ bool ordered() const { return false; }
    const int32_t *rp;
    const int32_t *col;
    int32_t M, nnz, G, first;
    const uint8_t *group_ok;
    __device__ __forceinline__ int32_t row(int64_t q) const { return static_cast<int32_t>(q); }
    __device__ __forceinline__ bool matched(int32_t r, int32_t &leader) const {
        const int32_t g = r < first ? 0 : 1 + (r - first) / G;
        int32_t end;
        unit_group_rows(g, G, first, M, leader, end);
        return group_ok[g] != 0;
    }
    __device__ __forceinline__ void run(int64_t q, int32_t &s, int32_t &e) const {
        const int32_t r = static_cast<int32_t>(q);
        int32_t leader;
        s = rp[r];
        e = matched(r, leader) && r != leader ? s : rp[r + 1];
    }
};

// pass 1: units of every tile; the grand total goes to pc->units
template <typename Runs>
__global__ void __launch_bounds__(kUnitBlock) k_unit_sums(Runs given, int64_t n, int32_t *__restrict__ tile_sums, PlanCounters *__restrict__ pc,
                                                          ListGate gate) {
    if (list_unused(gate, pc)) return;   // (nor will the list be)
    const auto runs = given.settled(pc);
    if constexpr (Runs::kChosen) {
        if (given.have_sums && runs.panels == 1) {   // (the grid may be a longer list's: no units in the tiles past this one's end)
            if (threadIdx.x == 0 && blockIdx.x * static_cast<int64_t>(unit_tile(runs.M)) >= runs.M) tile_sums[blockIdx.x] = 0;
            return;
        }
        n = static_cast<int64_t>(runs.panels) * runs.M;   // (at most the n that the grid was made for)
    }
    const int tile = unit_tile(n);
    const int64_t base = static_cast<int64_t>(blockIdx.x) * tile;
    int32_t local = 0;
    for (int k = threadIdx.x; k < tile; k += kUnitBlock)
        if (base + k < n) {
            int32_t s, e;
            runs.run(base + k, s, e);
            local += (e - s + 7) >> 3;
        }
    const int32_t total = block_sum(local);
    if (threadIdx.x == 0) {
        tile_sums[blockIdx.x] = total;
        if (total) atomicAdd(&pc->units, static_cast<unsigned long long>(total));
    }
}

// The units' copies of the S values, for lists in panels (unit_val null: they are made later, k_unit_values)
struct UnitValues {
    const float *s_val = nullptr;
    float *unit_val = nullptr;
};

// A list is ordered by size (k_unit_build) from one short row in this many on: with fewer the kernel gains nothing and building takes
// longer (5.2 M nonzeros in rows of 26: upload and run 247 us, 250 with the order).  Not where DRAM is the bound, see list_by_size.
constexpr unsigned kShortRowShare = 16;

// pass 2: the units of a tile.  HDR = int2 (plain units) or int4 (row groups).  scanned: tile_sums holds the units before each tile.
// BY_SIZE, plain units, where the row statistics bear it out: the tile's runs of 8 nonzeros or more come first, then the shorter ones, a
// unit each, from 7 nonzeros down to 1, so that the units of a warp step are of one size and the gather kernel can leave out the slots
// that none of them fills.  (Longer runs keep their units together: with their last ones sorted too, the units of a row are read by
// different SMs, and where DRAM is the bound, rows of 26 in two panels, K = 32 takes 540 us instead of 465.  A kernel of its own: with
// the order as an argument only, power-law panels of 36 M nonzeros take 454 us to build instead of 423.)
template <typename Runs, typename HDR, bool BY_SIZE>
__global__ void __launch_bounds__(kUnitBlock) k_unit_build(Runs given, int64_t n, const int32_t *__restrict__ tile_sums, int64_t cap,
                                                           PlanCounters *__restrict__ pc, HDR *__restrict__ units,
                                                           int32_t *__restrict__ unit_cols, bool scanned, ListGate gate, UnitValues values) {
    // enqueued before the host has seen the counters: nothing is written for a pattern that it is about to refuse, or for one
    // that will be computed otherwise
    if (list_unused(gate, pc) || !given.wanted(pc)) return;
    const auto runs = given.settled(pc);
    if constexpr (Runs::kChosen) n = static_cast<int64_t>(runs.panels) * runs.M;
    // (unsorted columns that the column scan has yet to find: the runs overlap, and the list is not used)
    if (pc->bad_row_ptr || pc->bad_coo || (runs.sorted() && gate.columns_scanned && pc->unsorted_cols)) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) pc->list_built = 1;
    // (rows of 1 .. 7 nonzeros)
    const bool by_size = BY_SIZE && runs.ordered() && kShortRowShare * (pc->hist[1] + pc->hist[2] + pc->hist[3]) >= pc->rows_nonempty;
    constexpr int kPerThread = kUnitTileMax / kUnitBlock;
    __shared__ int32_t first_unit[kUnitTileMax];   // of the tile's entries, relative to the tile
    __shared__ int32_t start[kUnitTileMax], length[kUnitTileMax];
    __shared__ int32_t of_size[8];                 // short runs of each length; then the first one's place
    __shared__ int32_t short_run[BY_SIZE ? kUnitTileMax : 1];   // their entries, by place
    const int tile = unit_tile(n);
    int64_t before = 0;
    if (scanned) {
        before = tile_sums[blockIdx.x];
    } else {
        int32_t part = 0;
        for (int i = threadIdx.x; i < static_cast<int>(blockIdx.x); i += kUnitBlock) part += tile_sums[i];
        before = block_sum(part);
    }
    const int64_t base = static_cast<int64_t>(blockIdx.x) * tile;
    const int per_thread = (tile + kUnitBlock - 1) / kUnitBlock;
    int32_t cnt[kPerThread], rank[kPerThread], local = 0;
    if (by_size) {
        if (threadIdx.x < 8) of_size[threadIdx.x] = 0;
        __syncthreads();
    }
#pragma unroll
    for (int k = 0; k < kPerThread; ++k) {
        cnt[k] = 0;
        const int i = threadIdx.x * per_thread + k;
        if (k >= per_thread || i >= tile) continue;
        int32_t s = 0, e = 0;
        if (base + i < n) runs.run(base + i, s, e);
        start[i] = s;
        length[i] = e - s;
        const bool is_short = by_size && e > s && e - s < 8;
        cnt[k] = is_short ? 0 : (e - s + 7) >> 3;
        local += cnt[k];
        if (is_short) rank[k] = atomicAdd(&of_size[e - s], 1);   // (their order has no effect on any result)
    }
    int32_t total;
    int32_t at = block_inclusive_scan(local, &total) - local;
    const int32_t in_order = total;
    if (by_size) {
        if (threadIdx.x == 0)
            for (int n = 7; n > 0; --n) {
                const int32_t c = of_size[n];
                of_size[n] = total;
                total += c;
            }
        if (threadIdx.x == 0) of_size[0] = total;
        __syncthreads();
        total = of_size[0];
    }
#pragma unroll
    for (int k = 0; k < kPerThread; ++k) {
        const int i = threadIdx.x * per_thread + k;
        if (k < per_thread && i < tile) {
            first_unit[i] = at;
            if (by_size && length[i] > 0 && length[i] < 8) short_run[of_size[length[i]] + rank[k] - in_order] = i;
        }
        at += cnt[k];
    }
    __syncthreads();
    if (before + total > cap) return;
    // four units at a time: the searches, then the loads, then the stores of all four are in flight together
    constexpr int kBatch = 4, kGroups = kUnitBlock / 8;
    const int slot = threadIdx.x & 7;
    const bool copy = values.unit_val && runs.sorted();
    for (int32_t u0 = threadIdx.x >> 3; u0 < total; u0 += kBatch * kGroups) {
        int32_t u[kBatch], entry[kBatch], first[kBatch], count[kBatch], c[kBatch];
        float v[kBatch];
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
            u[k] = min(u0 + k * kGroups, total - 1);
            entry[k] = 0;
        }
        // the entry that holds unit u: the last one that starts at or before it (tile: a power of two)
        for (int half = !BY_SIZE || u0 < in_order ? tile >> 1 : 0; half > 0; half >>= 1)
#pragma unroll
            for (int k = 0; k < kBatch; ++k)
                if (first_unit[entry[k] + half] <= u[k]) entry[k] += half;
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
            if (BY_SIZE && u[k] >= in_order) entry[k] = short_run[u[k] - in_order];
            const int32_t skip = BY_SIZE && u[k] >= in_order ? 0 : 8 * (u[k] - first_unit[entry[k]]);
            first[k] = start[entry[k]] + skip;
            count[k] = min(8, length[entry[k]] - skip);
            c[k] = runs.col[first[k] + min(slot, count[k] - 1)];
            if (copy) v[k] = values.s_val[first[k] + min(slot, count[k] - 1)];
        }
#pragma unroll
        for (int k = 0; k < kBatch; ++k) {
            if (u0 + k * kGroups >= total) break;
            if (unit_cols) unit_cols[8 * (before + u[k]) + slot] = c[k];
            if (copy) values.unit_val[8 * (before + u[k]) + slot] = v[k];
            if (slot == 0) {
                const int32_t row = runs.row(base + entry[k]);
                HDR h;
                h.x = first[k];
                h.y = row * 8 + (count[k] - 1);
                if constexpr (sizeof(HDR) == sizeof(int4)) {
                    int32_t leader;
                    h.z = length[entry[k]];
                    h.w = runs.matched(row, leader) ? runs.G : 1;
                }
                units[before + u[k]] = h;
            }
        }
    }
}

// units before range c of `parts` <= 8 row ranges, of a list over whole rows (whose tiles are in row order)
// (n_units < 0: as many as pc->units says)
__global__ void k_unit_cuts(const int2 *__restrict__ units, int32_t M, int32_t parts, int32_t n_units, PlanCounters *__restrict__ pc) {
    if (static_cast<int>(threadIdx.x) >= parts) return;
    const int32_t row = static_cast<int32_t>(range_start(M, threadIdx.x, parts));
    int64_t lo = 0, hi = n_units >= 0 ? n_units : static_cast<int64_t>(pc->units);
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if ((units[mid].y >> 3) < row) lo = mid + 1; else hi = mid;
    }
    pc->unit_cut[threadIdx.x] = static_cast<int>(lo);
}

// copies of the last unit up to a multiple of 8 (the bf16 kernel reads a step's 8 units as one block)
__global__ void k_unit_pad(int2 *__restrict__ units, int32_t *__restrict__ unit_cols, const PlanCounters *__restrict__ pc, int64_t cap) {
    const int64_t n = static_cast<int64_t>(pc->units);
    if (n == 0 || n > cap) return;
    const int64_t u = n + (threadIdx.x >> 3);
    if (u >= ((n + 7) & ~int64_t(7))) return;
    unit_cols[8 * u + (threadIdx.x & 7)] = unit_cols[8 * (n - 1) + (threadIdx.x & 7)];
    if ((threadIdx.x & 7) == 0) units[u] = units[n - 1];
}

// per-unit copies of the S values (column panels), one thread per slot: refreshed whenever S.val changes
__global__ void k_unit_values(const int2 *__restrict__ units, int32_t n_units, const float *__restrict__ s_val, float *__restrict__ usval) {
    for (int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; t < 8 * static_cast<int64_t>(n_units);
         t += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int2 u = units[t >> 3];
        usval[t] = s_val[u.x + min(static_cast<int>(t & 7), u.y & 7)];
    }
}

// ---- units over what the dense tiles left: runs of nonzeros whose bit in `covered` is clear -----------------------
// One warp per row, one word of the bitmap per lane; a run ends at the end of its word, so that words are independent.
__device__ __forceinline__ uint32_t uncovered_bits(const uint32_t *__restrict__ covered, int32_t word, int32_t a, int32_t b) {
    const int64_t first = 32 * static_cast<int64_t>(word);
    uint32_t bits = ~covered[word];
    if (first < a) bits &= ~0u << (a - first);
    if (first + 32 > b) bits &= ~0u >> (first + 32 - b);
    return bits;
}
// the next run of set bits: its start and length, taken out of `bits` (!= 0)
__device__ __forceinline__ int take_run(uint32_t &bits, int &start) {
    start = __ffs(bits) - 1;
    const uint32_t rest = ~(bits >> start);
    const int len = rest ? __ffs(rest) - 1 : 32;   // (rest = 0 only for a full word)
    bits = start + len >= 32 ? 0u : bits & (~0u << (start + len));
    return min(len, 32 - start);
}
__device__ __forceinline__ int run_units(uint32_t bits) {
    int n = 0, start;
    while (bits) n += (take_run(bits, start) + 7) >> 3;
    return n;
}
__global__ void k_residual_unit_count(const int32_t *__restrict__ rp, int32_t M, const uint32_t *__restrict__ covered, int32_t *__restrict__ counts) {
    const int lane = threadIdx.x & 31;
    const int64_t n_warps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
    for (int64_t r = (blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x) >> 5; r < M; r += n_warps) {
        const int32_t a = rp[r], b = rp[r + 1];
        int n = 0;
        if (b > a)
            for (int32_t w = (a >> 5) + lane; w <= (b - 1) >> 5; w += 32) n += run_units(uncovered_bits(covered, w, a, b));
        n = static_cast<int>(__reduce_add_sync(kFullMask, static_cast<unsigned>(n)));
        if (lane == 0) counts[r] = n;
    }
}
__global__ void k_residual_unit_fill(const int32_t *__restrict__ rp, int32_t M, const uint32_t *__restrict__ covered,
                                     const int32_t *__restrict__ offsets, const int32_t *__restrict__ col, int2 *__restrict__ units,
                                     int32_t *__restrict__ unit_cols) {
    const int lane = threadIdx.x & 31;
    const int64_t n_warps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
    for (int64_t r = (blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x) >> 5; r < M; r += n_warps) {
        const int32_t a = rp[r], b = rp[r + 1];
        if (b <= a) continue;
        int32_t off = offsets[r];
        const int32_t last = (b - 1) >> 5;
        for (int32_t w0 = a >> 5; w0 <= last; w0 += 32) {
            const int32_t w = w0 + lane;
            uint32_t bits = w <= last ? uncovered_bits(covered, w, a, b) : 0u;
            const int n = run_units(bits);
            const int32_t before = warp_inclusive_scan(n, lane);
            int32_t at = off + before - n;
            int start;
            while (bits) {
                const int len = take_run(bits, start);
                for (int skip = 0; skip < len; skip += 8, ++at) {
                    const int32_t first = 32 * w + start + skip, count = min(8, len - skip);
                    units[at] = make_int2(first, static_cast<int32_t>(r) * 8 + (count - 1));
#pragma unroll
                    for (int i = 0; i < 8; ++i) unit_cols[8 * static_cast<int64_t>(at) + i] = col[first + min(i, count - 1)];
                }
            }
            off += __shfl_sync(kFullMask, before, 31);
        }
    }
}

// ---- exclusive scan of int32 counts (three small kernels) -----------------------------------
// pass 1: sum of every tile of kScanTile values
__global__ void __launch_bounds__(kScanBlock) k_scan_tile_sums(const int32_t *__restrict__ v, int64_t n, int32_t *__restrict__ tile_sums) {
    const int64_t base = static_cast<int64_t>(blockIdx.x) * kScanTile + static_cast<int64_t>(threadIdx.x) * kScanPerThread;
    int32_t local = 0;
#pragma unroll
    for (int k = 0; k < kScanPerThread; ++k)
        if (base + k < n) local += v[base + k];
    int32_t total;
    block_inclusive_scan(local, &total);
    if (threadIdx.x == 0) tile_sums[blockIdx.x] = total;
}
// pass 2 (one block): exclusive scan of the tile sums in place; *grand_total = sum of everything
__global__ void __launch_bounds__(kScanBlock) k_scan_sums(int32_t *__restrict__ tile_sums, int32_t n_tiles, unsigned long long *__restrict__ grand_total) {
    int64_t carry = 0;
    for (int32_t base = 0; base < n_tiles; base += kScanBlock * kSumsPerThread) {
        const int32_t first = base + static_cast<int32_t>(threadIdx.x) * kSumsPerThread;
        int32_t v[kSumsPerThread], local = 0;
#pragma unroll
        for (int k = 0; k < kSumsPerThread; ++k) {
            v[k] = first + k < n_tiles ? tile_sums[first + k] : 0;
            local += v[k];
        }
        int32_t total;
        int32_t at = static_cast<int32_t>(carry) + block_inclusive_scan(local, &total) - local;
#pragma unroll
        for (int k = 0; k < kSumsPerThread; ++k) {
            if (first + k < n_tiles) tile_sums[first + k] = at;
            at += v[k];
        }
        carry += total;
    }
    if (threadIdx.x == 0) *grand_total = static_cast<unsigned long long>(carry);
}
// pass 3: exclusive scan inside every tile plus the tile's offset, in place
__global__ void __launch_bounds__(kScanBlock) k_scan_apply(int32_t *__restrict__ v, int64_t n, const int32_t *__restrict__ tile_offsets) {
    const int64_t base = static_cast<int64_t>(blockIdx.x) * kScanTile + static_cast<int64_t>(threadIdx.x) * kScanPerThread;
    int32_t x[kScanPerThread];
    int32_t local = 0;
#pragma unroll
    for (int k = 0; k < kScanPerThread; ++k) {
        x[k] = (base + k < n) ? v[base + k] : 0;
        local += x[k];
    }
    int32_t total;
    const int32_t inc = block_inclusive_scan(local, &total);
    int32_t run = tile_offsets[blockIdx.x] + inc - local;
#pragma unroll
    for (int k = 0; k < kScanPerThread; ++k) {
        if (base + k < n) v[base + k] = run;
        run += x[k];
    }
}

}  // namespace sddmm
