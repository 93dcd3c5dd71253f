// Upload-time kernels: validation of the uploaded pattern, the row-length
// histogram, COO -> row_ptr, the nnz-balanced work-item table and storage
// conversion.  They replace host loops of the reference
// (CSR::_dispatch, src/matrices/CSR.hpp:214-264; GPUPreprocessing::init_csr,
// src/competitors/gpu/gpu_preprocessing.hpp:56-128; gpu_convert_kernel,
// src/competitors/gpu/gpu_convert.cu:8-18) and run once per upload, outside
// the timed compute phase.
#pragma once

#include "device_utils.cuh"
#include "plan_sizes.cuh"
#include "../../include/sddmm_b200.h"

namespace sddmm {

struct PlanCounters {
    unsigned long long hist[SDDMM_B200_HIST_BINS];
    unsigned long long hist_nnz[SDDMM_B200_HIST_BINS];   // nonzeros held by the rows of each length bin
    unsigned long long rows_nonempty;
    unsigned long long cols_touched;
    unsigned long long dense_nnz;
    unsigned long long group_cover[9];   // nonzeros inside matching row groups: 2, 3, 4 rows per group x first full group at row 0 .. G-1
    int max_row_nnz;
    int bad_row_ptr;   // row_ptr not monotone / wrong ends
    int bad_col;       // column index outside [0, N)
    int unsorted_cols; // a column index smaller than its predecessor inside a row
    int dup_cols;      // a column index equal to its predecessor inside a row
    int bad_coo;       // COO row index out of range or decreasing
    int dense_tiles;
    int group_count[9];                  // matching row groups, same slots
    int residual_items;
    int unit_cut[8];                     // consumer: units before each of 8 equal row ranges
    unsigned long long units;            // row segments of the row-segment path
    unsigned long long window_nnz;       // nonzeros inside the selected 64x64 windows (summed per window)
    unsigned long long window_hint;      // nonzeros (estimate from every fourth one) whose 31st successor lies less than 64 columns ahead
    int block_samples;                   // sampled nonzeros that lie in what looks like a 64x64 block
    int n_anchors;                       // candidate origins of the arbitrary-offset tile detection
    int list_built;                      // 1: a list that was enqueued early has been written (see ListGate)
};

__device__ __forceinline__ int len_bin(int len) {
    if (len <= 0) return 0;
    int b = 32 - __clz(len);  // len in [2^(b-1), 2^b)
    return b < SDDMM_B200_HIST_BINS ? b : SDDMM_B200_HIST_BINS - 1;
}

constexpr int kUnitBlock = kPlanBlock;

// One tile of rows per block: monotonicity, histogram, max, nonempty count, row-start bits, and (tile_sums != nullptr) the
// units of the tile when every row is one run -- pass 1 of the plain unit list.
__global__ void __launch_bounds__(kUnitBlock) k_row_stats(const int32_t *__restrict__ rp, int32_t M, int64_t nnz, uint32_t *__restrict__ row_start_bits,
                                                          int32_t *__restrict__ tile_sums, PlanCounters *__restrict__ pc) {
    __shared__ unsigned int sh[SDDMM_B200_HIST_BINS];
    __shared__ unsigned long long sh_nnz[SDDMM_B200_HIST_BINS];
    __shared__ int s_max;
    if (threadIdx.x < SDDMM_B200_HIST_BINS) { sh[threadIdx.x] = 0; sh_nnz[threadIdx.x] = 0; }
    if (threadIdx.x == 0) s_max = 0;
    __syncthreads();
    int32_t units = 0;
    const int tile = unit_tile(M);
    for (int k = threadIdx.x; k < (tile + 31) / 32 * 32; k += kUnitBlock) {   // (whole warps)
        const int64_t i = blockIdx.x * static_cast<int64_t>(tile) + k;
        int len = -1;                                // no row, or one that is refused
        if (i < M && k < tile) {
            const int a = rp[i], b = rp[i + 1];
            if (b < a || a < 0 || b > nnz || (i == 0 && a != 0) || (i == M - 1 && b != nnz)) {
                pc->bad_row_ptr = 1;
            } else {
                len = b - a;
                units += (len + 7) >> 3;
                if (len > 0) atomicOr(&row_start_bits[a >> 5], 1u << (a & 31));
            }
        }
        // the rows of a warp share few length bins: one shared-memory update per bin and warp
        const unsigned live = __ballot_sync(kFullMask, len >= 0);
        if (len >= 0) {
            const int bin = len_bin(len);
            const unsigned same = __match_any_sync(live, bin);
            const unsigned lo = __reduce_add_sync(same, static_cast<unsigned>(len) & 0xffffu), hi = __reduce_add_sync(same, static_cast<unsigned>(len) >> 16);
            const int longest = __reduce_max_sync(same, len);
            if ((threadIdx.x & 31) == __ffs(same) - 1) {
                atomicAdd(&sh[bin], __popc(same));
                atomicAdd(&sh_nnz[bin], (static_cast<unsigned long long>(hi) << 16) + lo);
                atomicMax(&s_max, longest);
            }
        }
    }
    const int32_t total = block_sum(units);   // (a block-wide barrier)
    if (threadIdx.x == 0 && tile_sums) {
        tile_sums[blockIdx.x] = total;
        if (total) atomicAdd(&pc->units, static_cast<unsigned long long>(total));
    }
    if (threadIdx.x < SDDMM_B200_HIST_BINS && sh[threadIdx.x]) {
        atomicAdd(&pc->hist[threadIdx.x], (unsigned long long)sh[threadIdx.x]);
        if (sh_nnz[threadIdx.x]) atomicAdd(&pc->hist_nnz[threadIdx.x], sh_nnz[threadIdx.x]);
    }
    if (threadIdx.x == 0) {
        unsigned int nonempty = 0;
        for (int k = 1; k < SDDMM_B200_HIST_BINS; ++k) nonempty += sh[k];
        if (nonempty) atomicAdd(&pc->rows_nonempty, static_cast<unsigned long long>(nonempty));
        if (s_max) atomicMax(&pc->max_row_nnz, s_max);
    }
}

// Four nonzeros per thread: column range, distinct columns (one bit each), in-row ordering.  col is 16-byte aligned.
// LOCAL: the bits are collected per block in shared memory (columns up to kColScanLocalBytes * 8) and merged once at the
// end -- on the global bitmap every block that has not seen a bit yet updates it, and the updates of a popular word queue up
// (5.2 M nonzeros over 200 000 columns: 18 us, against 51 us with cached reads of the global bitmap and 102 us past L1).
constexpr int kColScanThreads = 1024;
constexpr int kColScanLocalBytes = 200 * 1024;
template <bool LOCAL>
__global__ void __launch_bounds__(kColScanThreads) k_col_scan(const int32_t *__restrict__ col, int64_t nnz, int32_t N, const uint32_t *__restrict__ row_start_bits,
                                                              uint32_t *__restrict__ touched, PlanCounters *__restrict__ pc) {
    extern __shared__ uint32_t seen[];
    const int words = static_cast<int>((static_cast<int64_t>(N) + 31) / 32);
    if (LOCAL) {
        for (int w = threadIdx.x; w < words; w += kColScanThreads) seen[w] = 0u;
        __syncthreads();
    }
    int32_t fresh = 0, dense = 0;
    bool bad = false, unsorted = false, dup = false;
    const int64_t stride = 4 * static_cast<int64_t>(gridDim.x) * kColScanThreads;
    for (int64_t j = 4 * (blockIdx.x * static_cast<int64_t>(kColScanThreads) + threadIdx.x); j < nnz; j += stride) {
        int c[5];
        const int n = static_cast<int>(min(static_cast<int64_t>(4), nnz - j));
        c[0] = j > 0 ? col[j - 1] : 0;
        if (n == 4) {
            const int4 q = *reinterpret_cast<const int4 *>(col + j);
            c[1] = q.x; c[2] = q.y; c[3] = q.z; c[4] = q.w;
        } else {
            for (int k = 0; k < 4; ++k) c[k + 1] = col[j + min(k, n - 1)];
        }
        if (j + 31 < nnz && static_cast<uint32_t>(col[j + 31] - c[1]) < 64u) dense += 4;   // (across a row boundary by chance only)
        const uint32_t starts = row_start_bits[j >> 5] >> (j & 31);   // (j is a multiple of 4: the four bits lie in one word)
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            if (c[k + 1] < 0 || c[k + 1] >= N) {
                bad = true;
            } else {
                uint32_t *word = (LOCAL ? seen : touched) + (c[k + 1] >> 5);
                const uint32_t bit = 1u << (c[k + 1] & 31);
                if (!(*word & bit)) {   // (a stale read only costs an update)
                    if (LOCAL) atomicOr(word, bit);
                    else if (!(atomicOr(word, bit) & bit)) ++fresh;
                }
            }
            if (k < n && !((starts >> k) & 1u) && (j > 0 || k > 0)) {
                unsorted |= c[k] > c[k + 1];
                dup |= c[k] == c[k + 1];
            }
        }
    }
    if (bad) pc->bad_col = 1;
    if (unsorted) pc->unsorted_cols = 1;
    if (dup) pc->dup_cols = 1;
    if (LOCAL) {
        __syncthreads();
        for (int w = threadIdx.x; w < words; w += kColScanThreads)
            if (seen[w]) fresh += __popc(seen[w] & ~atomicOr(&touched[w], seen[w]));
    }
    for (int o = 16; o > 0; o >>= 1) {
        fresh += __shfl_xor_sync(kFullMask, fresh, o);
        dense += __shfl_xor_sync(kFullMask, dense, o);
    }
    if ((threadIdx.x & 31) == 0 && fresh) atomicAdd(&pc->cols_touched, static_cast<unsigned long long>(fresh));
    if ((threadIdx.x & 31) == 0 && dense) atomicAdd(&pc->window_hint, static_cast<unsigned long long>(dense));
}

// COO (sorted by row) -> row_ptr.  Thread j owns the rows in (row[j-1], row[j]].  `base` is subtracted from every row index
// (a slice of a larger matrix that starts at row `base`).
__global__ void k_coo_to_row_ptr(const int32_t *__restrict__ row, int64_t nnz, int32_t M, int32_t base, int32_t *__restrict__ rp,
                                 PlanCounters *__restrict__ pc) {
    for (int64_t j = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; j <= nnz;
         j += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int64_t prev = (j == 0) ? -1 : static_cast<int64_t>(row[j - 1]) - base;
        const int64_t cur = (j == nnz) ? M : static_cast<int64_t>(row[j]) - base;
        if (prev < -1 || prev >= M || cur < 0 || cur > M || (j < nnz && cur >= M) || cur < prev) {
            pc->bad_coo = 1;
            continue;
        }
        for (int64_t r = prev + 1; r <= cur; ++r) rp[r] = static_cast<int32_t>(j);
    }
}

// one thread per work item: rows holding its first and last nonzero
__global__ void k_item_rows(const int32_t *__restrict__ rp, int32_t M, int64_t nnz, int32_t item_nnz, int32_t n_items,
                            int2 *__restrict__ item_rows) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n_items) return;
    const int64_t j0 = static_cast<int64_t>(t) * item_nnz;
    const int64_t j1 = min(nnz, j0 + item_nnz) - 1;
    int2 out;
    {
        int lo = 0, hi = M;
        while (hi - lo > 1) { const int mid = (lo + hi) >> 1; if (rp[mid] <= j0) lo = mid; else hi = mid; }
        out.x = lo;
    }
    {
        int lo = out.x, hi = M;
        while (hi - lo > 1) { const int mid = (lo + hi) >> 1; if (rp[mid] <= j1) lo = mid; else hi = mid; }
        out.y = lo;
    }
    item_rows[t] = out;
}

// ---- dense-tile detection (64x64 aligned tiles at least half full) -----------------------
// One warp per row: lanes take contiguous chunks of the (sorted) row so that runs of
// nonzeros inside one tile are counted locally and flushed with one atomic per run.
__global__ void k_tile_count(const int32_t *__restrict__ rp, const int32_t *__restrict__ col, int32_t M, int32_t tiles_per_row,
                             int32_t *__restrict__ counts) {
    const int64_t w = (blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (w >= M) return;
    const int a = rp[w], b = rp[w + 1];
    const int len = b - a;
    if (len == 0) return;
    const int per = (len + 31) >> 5;
    const int lo = a + lane * per, hi = min(b, lo + per);
    const int64_t base = static_cast<int64_t>(w >> 6) * tiles_per_row;
    int cur = -1, run = 0;
    for (int j = lo; j < hi; ++j) {
        const int t = col[j] >> 6;
        if (t != cur) {
            if (run) atomicAdd(&counts[base + cur], run);
            cur = t;
            run = 0;
        }
        ++run;
    }
    if (run) atomicAdd(&counts[base + cur], run);
}

// aligned tiles with >= min_count nonzeros: append their origin (first row, first column) to the dense list
__global__ void k_tile_select(const int32_t *__restrict__ counts, int64_t n_tiles, int32_t tiles_per_row, int32_t min_count,
                              int2 *__restrict__ origins, int32_t cap, PlanCounters *__restrict__ pc) {
    for (int64_t t = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; t < n_tiles;
         t += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        if (counts[t] >= min_count) {
            const int slot = atomicAdd(&pc->dense_tiles, 1);
            if (slot < cap) {
                origins[slot] = make_int2(static_cast<int32_t>(t / tiles_per_row) * 64, static_cast<int32_t>(t % tiles_per_row) * 64);
                atomicAdd(&pc->window_nnz, static_cast<unsigned long long>(counts[t]));
            }
        }
    }
}

// first position of [lo, hi) whose column is >= c (columns sorted inside a row)
__device__ __forceinline__ int32_t lower_col(const int32_t *__restrict__ col, int32_t lo, int32_t hi, int64_t c) {
    while (lo < hi) {
        const int32_t mid = (lo + hi) >> 1;
        if (col[mid] < c) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// ... the same by a whole warp: 32 probes per step, so a row of 1 000 nonzeros takes two dependent loads instead of ten
__device__ __forceinline__ int32_t warp_lower_col(const int32_t *__restrict__ col, int32_t lo, int32_t hi, int64_t c) {
    const int lane = threadIdx.x & 31;
    while (hi - lo > 32) {
        const int32_t step = (hi - lo) / 33 + 1;                 // probes at lo + step * (lane + 1) - 1: 33 pieces of at most `step`
        const int64_t at = lo + static_cast<int64_t>(step) * (lane + 1) - 1;
        const bool below = at < hi && col[at] < c;
        const int n = __popc(__ballot_sync(kFullMask, below));   // probes below c come first
        const int64_t end = lo + static_cast<int64_t>(step) * (n + 1) - 1;
        lo += step * n;
        hi = static_cast<int32_t>(min(static_cast<int64_t>(hi), end));
    }
    return lo + __popc(__ballot_sync(kFullMask, lo + lane < hi && col[lo + lane] < c));
}

// ---- dense 64x64 windows at ARBITRARY offsets ("randomly placed blocks") ---------------------------------------------
// Step 1, one warp per row: nonzero j is a CANDIDATE when at least `half` nonzeros of its row lie in the 64 columns
// that start at its own column.  One bit per nonzero; a warp takes the 32 nonzeros of one word at a time.
__global__ void k_window_candidates(const int32_t *__restrict__ rp, const int32_t *__restrict__ col, int32_t M, int32_t half,
                                    uint32_t *__restrict__ cand) {
    const int lane = threadIdx.x & 31;
    const int64_t n_warps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
    for (int64_t r = (blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x) >> 5; r < M; r += n_warps) {
        const int32_t a = rp[r], b = rp[r + 1];
        if (b - a < half) continue;
        for (int32_t j0 = a & ~31; j0 < b; j0 += 32) {
            const int32_t j = j0 + lane;
            // `half` nonzeros from j on fit into 64 columns <=> the (half-1)-th successor is closer than 64 columns
            const bool is = j >= a && j + half <= b && col[j + half - 1] - col[j] < 64;
            const uint32_t word = __ballot_sync(kFullMask, is);
            if (lane == 0 && word) atomicOr(&cand[j0 >> 5], word);   // (the first and the last word are shared with other rows)
        }
    }
}

// nonzeros of row r inside columns [c, c + 64)
__device__ __forceinline__ int32_t window_count(const int32_t *__restrict__ rp, const int32_t *__restrict__ col, int32_t r, int32_t c) {
    const int32_t a = rp[r], b = rp[r + 1];
    const int32_t lo = lower_col(col, a, b, c);
    return lower_col(col, lo, min(b, lo + 64), static_cast<int64_t>(c) + 64) - lo;
}

// Does the pattern hold 64x64 blocks at all?  One thread per sampled nonzero: it counts when `half` nonzeros of its row fit
// into the 64 columns from its own on AND the row 32 above or the row 32 below -- one of the two crosses the same block --
// has a sixth of the 64 columns around it.  Long rows alone (power-law patterns) fulfil the first, not the second.
__global__ void k_block_sample(const int32_t *__restrict__ rp, const int32_t *__restrict__ col, int32_t M, int64_t nnz, int32_t half, int32_t samples,
                               PlanCounters *__restrict__ pc) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    bool hit = false;
    if (t < samples) {
        // evenly spaced, plus a part of the step that differs from sample to sample
        const int64_t step = max(static_cast<int64_t>(1), nnz / samples);
        const int64_t at = static_cast<int64_t>(t) * nnz / samples + static_cast<int64_t>((static_cast<uint32_t>(t) * 2654435761u) % static_cast<uint64_t>(step));
        const int32_t j = static_cast<int32_t>(min(at, nnz - 1));
        if (j + half <= nnz && static_cast<uint32_t>(col[j + half - 1] - col[j]) < 64u) {
            int32_t lo = 0, hi = M;   // the row that holds j
            while (hi - lo > 1) {
                const int32_t mid = lo + (hi - lo) / 2;
                if (rp[mid] <= j) lo = mid; else hi = mid;
            }
            const int32_t c = col[j] - 31;
            auto crossed = [&](int32_t r) -> bool { return r >= 0 && r < M && window_count(rp, col, r, c) >= 11; };
            hit = j + half <= rp[lo + 1] && (crossed(lo - 32) || crossed(lo + 32));
        }
    }
    const unsigned all = __ballot_sync(kFullMask, hit);
    if ((threadIdx.x & 31) == 0 && all) atomicAdd(&pc->block_samples, __popc(all));
}

// Step 2, one warp per row: the row's candidates are cut greedily, left to right, into 64-column windows (a window
// starts at the first candidate at or after the end of the previous one), so every window of a row is visited once.  A
// window whose row above is NOT dense in the same columns is the top edge of a block and anchors a tile there -- and
// further tiles every 64 rows below it for as long as those rows stay dense in the same columns.  The cutting is serial,
// two loads per window; the windows are judged 32 at a time, one per lane.
__global__ void k_window_anchors(const int32_t *__restrict__ rp, const int32_t *__restrict__ col, int32_t M, int32_t half,
                                 const uint32_t *__restrict__ cand, int2 *__restrict__ anchors, int32_t cap, int *__restrict__ n_anchors) {
    const int lane = threadIdx.x & 31;
    // first candidate position in [j, b), or b
    auto next_cand = [&](int32_t j, int32_t b) -> int32_t {
        while (j < b) {
            const uint32_t word = cand[j >> 5] >> (j & 31);
            if (word) return min(b, j + __ffs(word) - 1);
            j = (j | 31) + 1;
        }
        return b;
    };
    const int64_t n_warps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
    for (int64_t r = (blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x) >> 5; r < M; r += n_warps) {
        const int32_t a = rp[r], b = rp[r + 1];
        if (b - a < half) continue;
        int32_t w = next_cand(a, b);
        while (w < b) {
            int32_t mine = -1;   // first column of this lane's window
            for (int k = 0; k < 32 && w < b; ++k) {
                const int32_t c0 = w + lane < b ? col[w + lane] : INT32_MAX, c1 = w + 32 + lane < b ? col[w + 32 + lane] : INT32_MAX;
                const int32_t c = __shfl_sync(kFullMask, c0, 0);
                if (lane == k) mine = c;
                const int inside = __popc(__ballot_sync(kFullMask, c0 - c < 64)) + __popc(__ballot_sync(kFullMask, c1 - c < 64));
                w = next_cand(w + inside, b);
            }
            if (mine >= 0 && (r == 0 || window_count(rp, col, static_cast<int32_t>(r) - 1, mine) < half)) {
                for (int32_t rr = static_cast<int32_t>(r); rr < M; rr += 64) {
                    if (rr != r && window_count(rp, col, rr, mine) < half) break;
                    const int slot = atomicAdd(n_anchors, 1);
                    if (slot < cap) anchors[slot] = make_int2(rr, mine);
                }
            }
            __syncwarp();
        }
    }
}

// Step 3, one thread per (anchor, row): nonzeros inside the anchored window, summed per anchor
__global__ void k_anchor_counts(const int32_t *__restrict__ rp, const int32_t *__restrict__ col, int32_t M, const int2 *__restrict__ anchors,
                                int32_t n_anchors, int32_t *__restrict__ counts) {
    const int64_t g = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (g >= static_cast<int64_t>(n_anchors) * 64) return;
    const int2 o = anchors[g >> 6];
    const int32_t row = o.x + static_cast<int32_t>(g & 63);
    int32_t n = row < M ? window_count(rp, col, row, o.y) : 0;
    for (int off = 16; off > 0; off >>= 1) n += __shfl_xor_sync(kFullMask, n, off);   // (64 rows of an anchor = 2 warps)
    if ((threadIdx.x & 31) == 0 && n) atomicAdd(&counts[g >> 6], n);
}
// Step 4: anchors whose window holds >= min_count nonzeros become dense tiles
__global__ void k_anchor_select(const int2 *__restrict__ anchors, const int32_t *__restrict__ counts, int32_t n_anchors, int32_t min_count,
                                int2 *__restrict__ origins, int32_t cap, PlanCounters *__restrict__ pc) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n_anchors || counts[t] < min_count) return;
    const int slot = atomicAdd(&pc->dense_tiles, 1);
    if (slot < cap) {
        origins[slot] = anchors[t];
        atomicAdd(&pc->window_nnz, static_cast<unsigned long long>(counts[t]));
    }
}

// Overlapping tiles (windows at arbitrary offsets): who computes a nonzero that lies in several of them is decided by a
// key, not by a race -- every (tile, row) proposes (row offset << 6 | column offset) for each of its nonzeros, the
// smallest key wins (two tiles that hold the same nonzero differ in their origin, hence in the key), so the same matrix
// always gets the same owners and the same tiles survive k_tile_keep.  owner: one word per nonzero, preset to ~0.
// One warp per (tile, row).
__global__ void k_tile_propose(const int32_t *__restrict__ rp, const int32_t *__restrict__ col, int32_t M, const int2 *__restrict__ origins,
                               int32_t n_dense, uint32_t *__restrict__ owner) {
    const int64_t g = (blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x) >> 5;
    if (g >= static_cast<int64_t>(n_dense) * 64) return;
    const int lane = threadIdx.x & 31, r = static_cast<int>(g & 63);
    const int2 o = origins[g >> 6];
    const int row = o.x + r;
    if (row >= M) return;
    const int end = rp[row + 1], start = warp_lower_col(col, rp[row], end, o.y);
#pragma unroll
    for (int h = 0; h < 2; ++h) {
        const int j = start + lane + 32 * h;
        const int c = j < end ? col[j] - o.y : 64;
        if (c < 64) atomicMin(&owner[j], (static_cast<uint32_t>(r) << 6) | static_cast<uint32_t>(c));
    }
}

// One warp per (dense tile, row): first CSR position of the row inside the tile's column range, presence mask of its 64
// columns, and the OWN mask -- the nonzeros this tile computes: all of them for tiles on the 64-grid, which never overlap
// (owner == nullptr), else what k_tile_propose gave them.  Owned nonzeros are marked in `covered` and credited to their
// work items.
template <typename Desc>
__global__ void k_tile_rows(const int32_t *__restrict__ rp, const int32_t *__restrict__ col, int32_t M, const int2 *__restrict__ origins,
                            int32_t n_dense, Desc *__restrict__ descs, uint32_t *__restrict__ covered, int32_t item_nnz,
                            int32_t *__restrict__ item_covered, int32_t *__restrict__ tile_owned, PlanCounters *__restrict__ pc,
                            const uint32_t *__restrict__ owner) {
    __shared__ int block_owned;
    if (threadIdx.x == 0) block_owned = 0;
    __syncthreads();
    const int64_t g = (blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (g < static_cast<int64_t>(n_dense) * 64) {
        const int t = static_cast<int>(g >> 6), r = static_cast<int>(g & 63);
        const int2 o = origins[t];
        const int row = o.x + r;
        int start = 0, owned = 0;
        uint32_t mask[2] = {0u, 0u}, own[2] = {0u, 0u};   // low and high word
        if (row < M) {
            const int end = rp[row + 1];
            start = warp_lower_col(col, rp[row], end, o.y);
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int j = start + lane + 32 * h;
                const int c = j < end ? col[j] - o.y : 64;
                const bool in = c < 64;
                const bool got = in && (!owner || owner[j] == ((static_cast<uint32_t>(r) << 6) | static_cast<uint32_t>(c)));
                const uint32_t bit = 1u << (c & 31);
                mask[0] |= __reduce_or_sync(kFullMask, in && c < 32 ? bit : 0u);
                mask[1] |= __reduce_or_sync(kFullMask, in && c >= 32 ? bit : 0u);
                own[0] |= __reduce_or_sync(kFullMask, got && c < 32 ? bit : 0u);
                own[1] |= __reduce_or_sync(kFullMask, got && c >= 32 ? bit : 0u);
                const unsigned live = __ballot_sync(kFullMask, got);
                owned += __popc(live);
                if (got) {
                    const unsigned word_peers = __match_any_sync(live, j >> 5);
                    const unsigned bits = __reduce_or_sync(word_peers, 1u << (j & 31));
                    if (lane == __ffs(word_peers) - 1) atomicOr(&covered[j >> 5], bits);
                    const unsigned item_peers = __match_any_sync(live, j / item_nnz);
                    if (lane == __ffs(item_peers) - 1) atomicAdd(&item_covered[j / item_nnz], __popc(item_peers));
                }
            }
        }
        if (lane == 0) {
            descs[t].start[r] = start;
            descs[t].mask[r] = (static_cast<unsigned long long>(mask[1]) << 32) | mask[0];
            descs[t].own[r] = (static_cast<unsigned long long>(own[1]) << 32) | own[0];
            if (owned) {
                atomicAdd(&tile_owned[t], owned);
                atomicAdd(&block_owned, owned);
            }
        }
    }
    __syncthreads();
    if (threadIdx.x == 0 && block_owned) atomicAdd(&pc->dense_nnz, static_cast<unsigned long long>(block_owned));
}

// Overlapping windows: a tile that ended up owning too few nonzeros (most of its window went to its neighbours) is not
// worth a job.  The tiles that own enough are copied to a second list, on which the ownership is then decided afresh.
__global__ void k_tile_keep(const int2 *__restrict__ origins, const int32_t *__restrict__ tile_owned, int32_t n_dense, int32_t min_owned,
                            int2 *__restrict__ kept, PlanCounters *__restrict__ pc) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n_dense || tile_owned[t] < min_owned) return;
    kept[atomicAdd(&pc->dense_tiles, 1)] = origins[t];
}

// work items that still hold nonzeros outside the dense tiles
__global__ void k_residual_items(const int32_t *__restrict__ item_covered, int32_t n_items, int32_t item_nnz, int64_t nnz,
                                 int32_t *__restrict__ item_ids, PlanCounters *__restrict__ pc) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n_items) return;
    const int64_t size = min(nnz, static_cast<int64_t>(t + 1) * item_nnz) - static_cast<int64_t>(t) * item_nnz;
    if (item_covered[t] < size) item_ids[atomicAdd(&pc->residual_items, 1)] = t;
}

// fp32-grade products from tf32 tensor cores: with hi = tf32(x), lo = tf32(x - hi),
//   a.b ~= a_lo*b_hi + a_hi*b_lo + a_hi*b_hi   (the dropped lo*lo term is ~2^-22 relative).
// The three products become ONE dot product of 3K-long rows:
//   first_operand = 1:  out row = [ lo | hi | hi ]     (used for A)
//   first_operand = 0:  out row = [ hi | lo | hi ]     (used for B)
__global__ void k_split_concat_tf32(const float *__restrict__ in, float *__restrict__ out, int64_t rows, int32_t K, int first_operand) {
    const int64_t n = rows * K;
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const float x = in[i];
        uint32_t h, l;
        asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(h) : "f"(x));
        const float hf = __uint_as_float(h);
        asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(l) : "f"(x - hf));
        const float lf = __uint_as_float(l);
        const int64_t r = i / K, k = i - r * K;
        float *o = out + r * 3 * K + k;
        o[0] = first_operand ? lf : hf;
        o[K] = first_operand ? hf : lf;
        o[2 * K] = hf;
    }
}

// rows of K floats -> rows of Ks floats (a multiple of 8), zero-padded; slice < Ks: slices of that many columns, all rows of one
// before the next.  specials (may be null): set to 1 when an element at or past column `last_part` is not finite.
__global__ void k_pad_rows(const float *__restrict__ in, float *__restrict__ out, int64_t rows, int32_t K, int32_t Ks, int32_t slice,
                           int32_t last_part, int32_t *__restrict__ specials) {
    const int32_t quads = Ks / 4;
    const int64_t n = rows * quads;
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n; i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int64_t r = i / quads;
        const int32_t k = 4 * static_cast<int32_t>(i - r * quads);
        const float *src = in + r * K + k;
        float4 v;
        v.x = k < K ? src[0] : 0.f;
        v.y = k + 1 < K ? src[1] : 0.f;
        v.z = k + 2 < K ? src[2] : 0.f;
        v.w = k + 3 < K ? src[3] : 0.f;
        if (specials && k >= last_part && !(isfinite(v.x) && isfinite(v.y) && isfinite(v.z) && isfinite(v.w))) *specials = 1;
        const int32_t part = k / slice;
        *reinterpret_cast<float4 *>(out + (part * rows + r) * slice + (k - part * slice)) = v;
    }
}

// bf16 storage: out = bf16(in) in rows of Ks >= K elements (zero-padded; K, Ks multiples of 4), and `in` keeps the rounded
// value (as fp32) for the tensor-core path.  specials, as above: of the rounded elements.
__global__ void k_f32_to_bf16(float *__restrict__ in, __nv_bfloat16 *__restrict__ out, int64_t rows, int32_t K, int32_t Ks, int32_t last_part,
                              int32_t *__restrict__ specials) {
    const int32_t quads = Ks / 4;
    const int64_t n = rows * quads;
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n; i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int64_t r = i / quads;
        const int32_t k = 4 * static_cast<int32_t>(i - r * quads);
        uint2 packed = make_uint2(0u, 0u);
        if (k < K) {
            float4 *src = reinterpret_cast<float4 *>(in + r * K + k);
            const float4 v = *src;
            const __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
            packed = make_uint2(*reinterpret_cast<const uint32_t *>(&lo), *reinterpret_cast<const uint32_t *>(&hi));
            const float4 r = make_float4(__low2float(lo), __high2float(lo), __low2float(hi), __high2float(hi));
            *src = r;
            if (specials && k >= last_part && !(isfinite(r.x) && isfinite(r.y) && isfinite(r.z) && isfinite(r.w))) *specials = 1;
        }
        reinterpret_cast<uint2 *>(out)[i] = packed;
    }
}

}  // namespace sddmm
