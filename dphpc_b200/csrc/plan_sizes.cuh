// Sizes that the planner and its kernels agree on.  Plain arithmetic, compiled for the host alone too.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

namespace sddmm {

// Unit lists (unit_plan.cuh) are scanned in tiles of this many entries: small tiles for short lists, so that every SM has
// several blocks to build (200 000 rows: 113 us in 196 blocks of 1024 entries), larger ones for long lists.
constexpr int kUnitTileMax = 1024;
__host__ __device__ __forceinline__ int unit_tile(int64_t n) { return n > (1 << 20) ? kUnitTileMax : n > (1 << 18) ? 256 : 128; }
// first of `parts` row ranges' rows, on a tile of the list over whole rows
__host__ __device__ __forceinline__ int64_t range_start(int64_t M, int c, int parts) { return c >= parts ? M : M * c / parts / unit_tile(M) * unit_tile(M); }
inline int64_t unit_tiles(int64_t n) { return (n + unit_tile(n) - 1) / unit_tile(n); }

// A block of the list's second kernel adds up the sums of all tiles before its own, which is quadratic in their number: fine for a few
// thousand (a launch between the two kernels costs more), 0.6 GB of loads for 17 800, a terabyte for the 786 000 of 2^28 rows in
// three panels.  From here on one block scans the sums first.
constexpr int kDirectTiles = 4096;

// ... and the residual lists' row counts in tiles of
constexpr int kScanBlock = 256;
constexpr int kScanPerThread = 8;
constexpr int kScanTile = kScanBlock * kScanPerThread;
constexpr int kSumsPerThread = 16;   // ... and their sums in steps of this many per thread of one block
inline int64_t scan_tiles(int64_t n) { return (n + kScanTile - 1) / kScanTile; }

// Tile sums that a plan may need: whole rows, plain column panels, panels for the long rows with the short rows as one more
// entry (panels_long = 0: no candidate), residual rows.  The row statistics choose among the forms after the memory has been
// laid out, and a longer list can have FEWER tiles than a shorter one (1.2 M entries 1172, 600 000 entries 2344), so every
// form counts by itself.
inline int64_t plan_tile_sums(int64_t M, int64_t panels_plain, int64_t panels_long) {
    int64_t tiles = std::max(unit_tiles(M), scan_tiles(M));
    tiles = std::max(tiles, unit_tiles(M * std::max<int64_t>(1, panels_plain)));
    if (panels_long > 0) tiles = std::max(tiles, unit_tiles(M * (panels_long + 1)));
    return tiles;
}

// Units of a list of `runs` runs (at most one per row, nonempty) that hold `nnz` nonzeros: a run of L takes at most L / 8 + 7 / 8.
// The residual lists, whose runs also end at every 32nd nonzero, stay below it too.  The end of a row inside a word costs two
// partial units that together waste 8 slots or none; a row's cut by the window of a dense tile costs two that waste at most 14, and a
// tile cuts at most 64 rows but owns 1024 nonzeros or more (k_tile_keep), which take no units: 64 * 14 / 8 = 112 against 1024 / 8.
constexpr int kTileMinOwned = 1024;
inline int64_t unit_capacity(int64_t nnz, int64_t runs) { return nnz / 8 + runs + 8; }

// Elements from one row of A or B to the next for the row-segment kernels.  Rows start on a 128-byte line (short rows: do
// not cross one), so that a piece of a row is one line: with rows of 200 bytes back to back a piece touches two, and K = 50
// takes longer than K = 64 (64 against 46 us for 2.4 M nonzeros).
inline int64_t padded_row(bool bf16, int64_t K) {
    const int64_t line = bf16 ? 64 : 32;
    if (K > 256) return (K + 63) / 64 * 64;
    if (4 * K <= line) return line / 4;
    if (2 * K <= line) return line / 2;
    return (K + line - 1) / line * line;
}
// ... and without copies of A and B in that form: fp32 rows as they are, where they are whole 32-byte parts (0: not possible)
inline int64_t unpadded_row(int64_t K) { return K % 8 == 0 && K <= 256 ? K : 0; }

// What fills L2 in effect: a line that is read by SMs of both dies is kept in both halves of L2, so gathers at random begin to miss in a
// table of half its size, and from 0.85 times its size on the misses cost more than panels do.
constexpr double kPanelsFrom = 0.85;

// Whether the short runs of a list lie side by side (k_unit_build): for the fp32 kernels, which then leave out empty slots (the bf16
// kernel loads a unit at a time; those for rows of three pieces, and for panels of an odd number of them, load all slots), where the
// gathers hit L2 or only long rows are cut into panels.  Poisson rows of 8, B 262 MB, K = 128 265 -> 273 us with the order, K = 256
// 245 -> 260.  row: elements of a row of B that one launch takes; gathered: bytes of B it gathers from; l2 <= 0: not known.
inline bool by_size(bool bf16, int64_t row, bool long_rows, double gathered, double l2) {
    const int64_t pieces = (row + 31) / 32;
    if (bf16 || row < 32 || pieces == 3 || (long_rows && pieces > 1 && pieces % 2 == 1)) return false;
    return long_rows || l2 <= 0 || gathered <= kPanelsFrom * l2;
}

}  // namespace sddmm
