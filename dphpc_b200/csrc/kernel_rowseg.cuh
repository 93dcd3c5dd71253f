// Row-segment SDDMM kernels: the general path for short, long and power-law rows.
//
// Work decomposition (no atomics, exactly one writer per nonzero): every row is cut into SEGMENTS of at most 8
// consecutive nonzeros.  The list of segments ("units": first CSR position, row, count) and a copy of each unit's 8
// column indices are built once per upload on the device (unit_plan.cuh), so the kernels search nothing and stage
// nothing -- they are one streaming loop, grid-stride, balanced whatever the row-length distribution.
//
// A warp step takes 8 consecutive units, one per group of 4 lanes.  A row of A or B is read in PIECES of 128 bytes: lane t
// of a group holds bytes [32t, 32t + 32) of the piece in one 256-bit load, so one load instruction fetches the same piece
// of 8 B rows (one per unit), and the A piece in registers serves the unit's 8 nonzeros.  The loop is ROLLING: as soon as
// the B piece of slot i has been multiplied, its registers are given to the piece that slot needs next (the next piece of
// the same units, or the first one of the next units), so a warp has up to 8 loads of 1 KB in flight all the time; unit headers
// and column indices run one to two steps ahead, the A piece one stage ahead.  Every load is in range (a slot past a segment's
// end repeats its last nonzero, a group past the list's end the last unit).  Two neighbouring slots that no unit of a step fills
// are left out by the whole warp (see most_slots): their registers keep what an earlier step or the first one, which loads all
// slots, has put there, a slot's sum is made of its own registers only, and sums of slots past a unit's count are never stored.
//
// What bounds it: per nonzero one B row crosses from L2 to the SM (random 128-byte rows that hit L2: at most 153 G rows/s
// measured, 64 bytes per clock and SM) and, where B does not fit L2, comes from HBM.  37.5 M nonzeros, K = 32, B in L2:
// 294 us = 18.6 TB/s, against 347-365 us for a form with 16-byte chunks on groups of 8 lanes, which issues twice the loads
// and four times the instructions per nonzero.
//
// Column panels: when B is much larger than the L2 cache the unit list is built PANEL-MAJOR -- the columns are cut into P
// panels, a row contributes one run of segments per panel it touches, and all segments of panel 0 come before those of
// panel 1 and so on.  All CTAs walk the list in step, so the gathers of a panel find most of their B rows in L2.  (Rows of A
// are asked to leave L2 first, see ld_piece_first; asking it to keep the gathered rows of B adds nothing: measured.)
#pragma once

#include "device_utils.cuh"

namespace sddmm {

// unit.x = CSR position of the first nonzero of the segment; unit.y = row * 8 + (count - 1)
constexpr int kUnitRowLimit = 1 << 28;   // rows the encoding can name
constexpr int64_t kUnitLimit = (int64_t(1) << 31) - (int64_t(1) << 22);   // units a list may hold: step arithmetic stays in 32 bits

struct RowSegArgs {
    const int2 *units;         // n_units (> 0), padded to a multiple of 8 with copies of the last one
    const int32_t *unit_cols;  // 8 column indices per unit (slots past the count repeat the last one)
    const float *s_val;        // nnz values in CSR order, or (COPIES) 8 per unit in list order
    float *p_val;              // nnz
    const void *A;             // rows row_stride bytes apart, 32-byte aligned
    const void *B;
    int32_t n_units;
    uint32_t row_stride;       // bytes, a multiple of 32
    int32_t row_bytes;         // bytes of a row that this launch covers (a multiple of 32)
    float one;                 // 1
};

constexpr int kRowSegWarps = 8;
constexpr int kSlotStep = 2;   // slots that are loaded or left out together (see most_slots)

// ---- 256-bit loads (32-byte aligned) and packed fp32 arithmetic ------------------------------------------------------
// (volatile: the order in which the loads are written is the order of the rolling loop)
struct Piece {
    float2 v[4];
};
struct Cols8 {
    int32_t v[8];
};
__device__ __forceinline__ Piece ld_piece(const unsigned char *p) {
    Piece r;
    asm volatile("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(r.v[0].x), "=f"(r.v[0].y), "=f"(r.v[1].x), "=f"(r.v[1].y), "=f"(r.v[2].x), "=f"(r.v[2].y), "=f"(r.v[3].x),
                   "=f"(r.v[3].y)
                 : "l"(p));
    return r;
}
// ... of A: used by one or two units, then not again before the rest of A has passed through, so it is the first to leave L2 and
// B's rows stay.  20 M nonzeros in rows of 20, B 128 / 256 MB in panels: K = 32 271 -> 256 us, K = 64 567 -> 525; 37.5 M, rows of 26,
// K = 32 511 -> 500, bf16 K = 128 1135 -> 1096.  (evict_last on the gathers of B adds nothing.)
__device__ __forceinline__ Piece ld_piece_first(const unsigned char *p) {
    Piece r;
    asm volatile("ld.global.nc.L2::evict_first.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(r.v[0].x), "=f"(r.v[0].y), "=f"(r.v[1].x), "=f"(r.v[1].y), "=f"(r.v[2].x), "=f"(r.v[2].y), "=f"(r.v[3].x),
                   "=f"(r.v[3].y)
                 : "l"(p));
    return r;
}
// ... that has L2 fetch the whole 256-byte block it lies in: the first of two pieces of a row that are wanted one after the other
__device__ __forceinline__ Piece ld_piece_of_two(const unsigned char *p) {
    Piece r;
    asm volatile("ld.global.nc.L2::256B.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=f"(r.v[0].x), "=f"(r.v[0].y), "=f"(r.v[1].x), "=f"(r.v[1].y), "=f"(r.v[2].x), "=f"(r.v[2].y), "=f"(r.v[3].x),
                   "=f"(r.v[3].y)
                 : "l"(p));
    return r;
}
__device__ __forceinline__ void prefetch_l2(const void *p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
// (read once: first to leave L2 as well, 37.5 M nonzeros, rows of 26, K = 32 478 -> 465 us)
__device__ __forceinline__ Cols8 ld_cols(const int32_t *p) {
    Cols8 r;
    asm volatile("ld.global.nc.L1::no_allocate.L2::evict_first.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r.v[0]), "=r"(r.v[1]), "=r"(r.v[2]), "=r"(r.v[3]), "=r"(r.v[4]), "=r"(r.v[5]), "=r"(r.v[6]), "=r"(r.v[7])
                 : "l"(p));
    return r;
}
// two IEEE fused multiply-adds in one instruction
__device__ __forceinline__ float2 fma2(const float2 &a, const float2 &b, const float2 &c) {
    float2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;"
        : "=l"(reinterpret_cast<unsigned long long &>(d))
        : "l"(reinterpret_cast<const unsigned long long &>(a)), "l"(reinterpret_cast<const unsigned long long &>(b)),
          "l"(reinterpret_cast<const unsigned long long &>(c)));
    return d;
}
__device__ __forceinline__ float dot_piece(const Piece &a, const Piece &b, float acc) {
    float2 s = make_float2(acc, 0.f);
#pragma unroll
    for (int k = 0; k < 4; ++k) s = fma2(a.v[k], b.v[k], s);
    return s.x + s.y;
}
// What the lanes past the end of a row's last piece read in place of A.  They are sent here by their address: clearing the
// registers after the load would make every warp wait for it on the spot.
__device__ __align__(32) const float g_zero_part[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
__device__ __forceinline__ const unsigned char *row_at(const unsigned char *base, int32_t row, uint32_t stride) {
    return base + static_cast<uint64_t>(static_cast<uint32_t>(row)) * stride;
}

// Sum 8 per-lane values over the 4 lanes of a group: lane t ends up with the sums of slots t and t + 4.  (The additions of
// a slot are the same ones whatever its position, so a nonzero's value does not depend on how its row was cut.)
__device__ __forceinline__ float2 group4_transpose_reduce(const float (&a)[8], int t) {
    float w[4];
    const bool odd = (t & 1) != 0, high = (t & 2) != 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {   // w[i]: slot 2i + (t & 1)
        const float send = odd ? a[2 * i] : a[2 * i + 1];
        const float keep = odd ? a[2 * i + 1] : a[2 * i];
        w[i] = keep + __shfl_xor_sync(kFullMask, send, 1);
    }
    float2 r;
    r.x = (high ? w[1] : w[0]) + __shfl_xor_sync(kFullMask, high ? w[0] : w[1], 2);
    r.y = (high ? w[3] : w[2]) + __shfl_xor_sync(kFullMask, high ? w[2] : w[3], 2);
    return r;
}

// K in slices, one launch each: P.val carries the sum so far, and S comes in once, with the last slice -- a product per slice would
// make Inf - Inf of a large or infinite S value where the whole sum has a value, and reads S once per slice.  (The earlier slices
// multiply by args.one all the same: without the instruction the compiler spills in the first slice, K = 128 256 -> 265 us.)
enum SliceStep : int { kWholeRows, kFirstSlice, kNextSlice, kLastSlice };
__device__ __forceinline__ constexpr bool step_adds(int step) { return step == kNextSlice || step == kLastSlice; }
__device__ __forceinline__ constexpr bool step_scales(int step) { return step == kWholeRows || step == kLastSlice; }
template <int STEP>
__device__ __forceinline__ float step_value(float dot, float p, float s) {
    return (step_adds(STEP) ? p + dot : dot) * s;
}

// Whether some lanes of a row's last piece lie past its end: never (whole pieces: no addresses and registers for them), such lanes
// multiply zeros, or they leave the product out.  Without the logic: 6 M nonzeros, K = 128 220 -> 215 us, 3 M, K = 256 213 -> 190; bf16,
// K = 128, 37.5 M 1117 -> 1067, K = 32, 5.2 M 55 -> 44.  It stays where the kernel is slower without: for B beyond L2 (one form, its
// registers spill), rows of three pieces (K = 96: 44 against 46 us), bf16 rows of 64 (10 M: 109 against 123) and bf16 rows of 32 in
// panels (power law, 36 M: 349 against 358; Poisson rows of 30, 65 M: 696 against 721).
enum RowTail : int { kNoTail, kTail, kTailSpecials };

// How many stages before its load a piece of A is asked into L2.  A row of A is used by one or two units and comes from HBM,
// whose latency under load is longer than a stage: 9 M nonzeros, B in L2, K = 256: 880 us without, 725 with (K = 64 185 -> 168,
// K = 128 351 -> 325).  The best distances, measured, are 1, 3 and 2 for up to 2, 4 and more pieces; a prefetch of the whole row
// two steps ahead takes too much of L2 (K = 256 950 us).
__host__ __device__ constexpr int a_prefetch_stages(int pieces) { return pieces <= 2 ? 1 : pieces <= 4 ? 3 : 2; }

// fp32 rows of NP pieces.  (From NP = 3 on the 128 registers do not quite hold the loop, a few words of it are spilled; with the
// registers of one CTA per SM it is 20 % slower.)  The last piece may be partial: the lanes past its end
// read the row's last 32 bytes once more and multiply them by zero.  SPECIALS: such lanes leave the product out, as a factor of
// zero does not where B holds an infinity (0 x Inf is NaN).  Rows of one piece always do (K = 16: 335 against 336 us); longer ones only where a conversion of B has seen a non-finite
// element in the last 32 bytes of a row, since it costs registers that the rolling loop wants (ragged last piece, in L2, K = 33 /
// 50 / 100: 84 / 46.7 / 110 us without, 89 / 47.8 / 115 with it; zeros read in place of B: 105 / 55 / 114).  COPIES:
// S values come from per-unit copies in list order (column panels: a run is a short piece of its row, whose sectors two or more panel
// passes would read in turn).  STEP: which part of the dot products this launch adds up.
// (All index arithmetic of the loop is 32-bit: with 64-bit selects the compiler splits the loop body and the rolling is
// lost, 488 -> 574 us.  NP is a compile-time number for the same reason.)
template <int NP, int TAIL, bool COPIES, int STEP>
__global__ void __launch_bounds__(kRowSegWarps * 32, 2) sddmm_rowseg_kernel(const RowSegArgs args) {
    const int lane = threadIdx.x & 31;
    const int t = lane & 3;        // 32-byte part of a piece
    const int grp = lane >> 2;     // which of the warp's 8 units
    const int n_steps = (args.n_units + 7) >> 3;
    const int n_warps = static_cast<int>(gridDim.x) * kRowSegWarps;
    int b = static_cast<int>(blockIdx.x) * kRowSegWarps + (threadIdx.x >> 5);
    if (b >= n_steps) return;
    const int last_unit = args.n_units - 1;
    constexpr bool SPECIALS = TAIL == kTailSpecials;
    const bool off = TAIL != kNoTail && 128 * (NP - 1) + 32 * t >= args.row_bytes;   // this lane's part of the last piece lies past the row
    const uint32_t stride = args.row_stride;
    const unsigned char *At = static_cast<const unsigned char *>(args.A) + 32 * t;
    const unsigned char *Bt = static_cast<const unsigned char *>(args.B) + 32 * t;
    const int o_last = off ? args.row_bytes - 32 - 32 * t : 128 * (NP - 1);   // (such a lane reads the row's last 32 bytes)

    auto unit_index = [&](int step) -> int { const int u = 8 * step + grp; return u < last_unit ? u : last_unit; };
    auto load_unit = [&](int step) -> int2 { return __ldcs(args.units + unit_index(step)); };
    auto load_cols = [&](int step) -> Cols8 { return ld_cols(args.unit_cols + 8 * static_cast<int64_t>(unit_index(step))); };
    // The slots that any unit of a step fills.  Short runs lie side by side in the list, by length (unit_plan.cuh), so where rows are
    // short whole steps have few; the loads of the others are left out (their sums come from old registers and are not stored).
    // Power-law rows, K = 32: 5 M nonzeros 66 -> 60 us, 36 M 428 -> 402; Poisson rows of 10 48 -> 45.  One slot at a time
    // 396 us, but K = 128 in L2 100 against 95; loads that depend on their own lane's count serialise the loop.
    // Not for rows of one ragged piece (0.5 M nonzeros, K = 16 15.6 against 18 us), nor of three pieces and panels of rows of an odd
    // number, which the compiler does not roll with the branches in (K = 96, panels, 9 M nonzeros 286 -> 349 us, 52 000 13 -> 15).
    constexpr bool kLeaveOut = NP != 3 && !(NP == 1 && TAIL == kTailSpecials) && !(COPIES && NP > 1 && NP % 2 == 1);
    auto most_slots = [&](const int2 &u) -> int { return static_cast<int>(__reduce_max_sync(kFullMask, static_cast<unsigned>(u.y) & 7u)) + 1; };
    auto piece_offset = [&](int p) -> int { return p == NP - 1 ? o_last : 128 * p; };
    auto load_a = [&](int row, int p) -> Piece {
        const unsigned char *q = row_at(At + piece_offset(p), row, stride);
        return ld_piece_first(p == NP - 1 && off ? reinterpret_cast<const unsigned char *>(g_zero_part) : q);
    };

    int2 un = load_unit(b), un_next = load_unit(b + n_warps);
    Cols8 cols = load_cols(b);
    Piece a = load_a(un.y >> 3, 0), bq[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) bq[i] = ld_piece(row_at(Bt + piece_offset(0), cols.v[i], stride));
    int slots = kLeaveOut ? most_slots(un) : 8;   // of the step
    Cols8 cols_next = load_cols(b + n_warps);

    while (true) {
        const int next = b + n_warps;
        const int count = 8 * b + grp <= last_unit ? (un.y & 7) : -1;
        // S values of the slots this lane will write (t and t + 4), requested before the gathers
        const float *sv = COPIES ? args.s_val + 8 * static_cast<int64_t>(unit_index(b)) : args.s_val + un.x;
        const float s0 = step_scales(STEP) ? __ldcs(sv + (COPIES ? t : min(t, un.y & 7))) : args.one;
        const float s1 = step_scales(STEP) ? __ldcs(sv + (COPIES ? t + 4 : min(t + 4, un.y & 7))) : args.one;
        float p0 = 0.f, p1 = 0.f;
        if (step_adds(STEP) && t <= count) p0 = __ldcs(args.p_val + un.x + t);
        if (step_adds(STEP) && t + 4 <= count) p1 = __ldcs(args.p_val + un.x + t + 4);
        const int2 un_next2 = load_unit(next + n_warps);
        const Cols8 cols_next2 = load_cols(next + n_warps);

        const int slots_next = kLeaveOut ? most_slots(un_next) : 8;
        float acc[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] = 0.f;
#pragma unroll
        for (int p = 0; p < NP; ++p) {
            const bool last = p == NP - 1;
            const int p_next = last ? 0 : p + 1;
            const Piece a_next = load_a((last ? un_next.y : un.y) >> 3, p_next);
            constexpr int kAhead = a_prefetch_stages(NP);
            const int pf = p + 1 + kAhead;   // ... and the A piece kAhead stages after that one, to L2
            if (t == 0) prefetch_l2(row_at(static_cast<const unsigned char *>(args.A) + 128 * (pf % NP), (pf < NP ? un.y : pf < 2 * NP ? un_next.y : un_next2.y) >> 3, stride));
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float sum = dot_piece(a, bq[i], acc[i]);
                acc[i] = SPECIALS && last && off ? acc[i] : sum;
                if (!kLeaveOut || i / kSlotStep * kSlotStep < (last ? slots_next : slots)) {   // warp-uniform
                    const unsigned char *q = row_at(Bt + piece_offset(p_next), last ? cols_next.v[i] : cols.v[i], stride);
                    bq[i] = NP > 1 && p_next % 2 == 0 ? ld_piece_of_two(q) : ld_piece(q);
                }
            }
            a = a_next;
        }
        const float2 dot = group4_transpose_reduce(acc, t);
        if (t <= count) __stcs(args.p_val + un.x + t, step_value<STEP>(dot.x, p0, s0));
        if (t + 4 <= count) __stcs(args.p_val + un.x + t + 4, step_value<STEP>(dot.y, p1, s1));

        if (next >= n_steps) break;   // warp-uniform
        b = next;
        un = un_next;
        slots = slots_next;
        un_next = un_next2;
        cols = cols_next;
        cols_next = cols_next2;
    }
}

// The same for whole rows (NP even) of a B that does not fit L2 and is gathered without column panels: DRAM is the
// bound, and it likes few rows open at a time.  The stages go through all pieces of 4 slots, two pieces of 128 bytes at a
// time, before the other 4: half the rows in flight, twice the bytes of each.  9 M nonzeros in rows of 13, B 358 / 717 MB:
// K = 128 697 -> 638 us, K = 256 1581 -> 1559; 13 M nonzeros in rows of 9, B 373 MB: K = 64 558 -> 524; with B in L2 the order above is
// faster (K = 128 385 against 414).
template <int NP, bool SPECIALS, int STEP>
__global__ void __launch_bounds__(kRowSegWarps * 32, 2) sddmm_rowseg_wide_kernel(const RowSegArgs args) {
    const int lane = threadIdx.x & 31;
    const int t = lane & 3;
    const int grp = lane >> 2;
    const int n_steps = (args.n_units + 7) >> 3;
    const int n_warps = static_cast<int>(gridDim.x) * kRowSegWarps;
    int b = static_cast<int>(blockIdx.x) * kRowSegWarps + (threadIdx.x >> 5);
    if (b >= n_steps) return;
    const int last_unit = args.n_units - 1;
    const bool off = 128 * (NP - 1) + 32 * t >= args.row_bytes;   // this lane's part of the last piece lies past the row
    const uint32_t stride = args.row_stride;
    const unsigned char *At = static_cast<const unsigned char *>(args.A) + 32 * t;
    const unsigned char *Bt = static_cast<const unsigned char *>(args.B) + 32 * t;
    const int o_last = off ? args.row_bytes - 32 - 32 * t : 128 * (NP - 1);
    constexpr int kPairs = NP / 2;

    auto unit_index = [&](int step) -> int { const int u = 8 * step + grp; return u < last_unit ? u : last_unit; };
    auto load_unit = [&](int step) -> int2 { return __ldcs(args.units + unit_index(step)); };
    auto load_cols = [&](int step) -> Cols8 { return ld_cols(args.unit_cols + 8 * static_cast<int64_t>(unit_index(step))); };
    auto piece_offset = [&](int p) -> int { return p == NP - 1 ? o_last : 128 * p; };
    auto load_a = [&](Piece (&a)[2], int row, int q) {
        const unsigned char *r = row_at(At, row, stride);
        a[0] = ld_piece_first(r + piece_offset(2 * q));
        a[1] = ld_piece_first(2 * q + 1 == NP - 1 && off ? reinterpret_cast<const unsigned char *>(g_zero_part) : r + piece_offset(2 * q + 1));
    };
    auto load_b = [&](Piece (&x)[2], int col, int q) {
        const unsigned char *r = row_at(Bt, col, stride);
        x[0] = ld_piece(r + piece_offset(2 * q));
        x[1] = ld_piece(r + piece_offset(2 * q + 1));
    };

    int2 un = load_unit(b), un_next = load_unit(b + n_warps);
    Cols8 cols = load_cols(b);
    Piece a[2], bq[4][2];
    load_a(a, un.y >> 3, 0);
#pragma unroll
    for (int i = 0; i < 4; ++i) load_b(bq[i], cols.v[i], 0);

    while (true) {
        const int next = b + n_warps;
        const int count = 8 * b + grp <= last_unit ? (un.y & 7) : -1;
        const float *sv = args.s_val + un.x;
        const float s0 = step_scales(STEP) ? __ldcs(sv + min(t, un.y & 7)) : args.one;
        const float s1 = step_scales(STEP) ? __ldcs(sv + min(t + 4, un.y & 7)) : args.one;
        float p0 = 0.f, p1 = 0.f;
        if (step_adds(STEP) && t <= count) p0 = __ldcs(args.p_val + un.x + t);
        if (step_adds(STEP) && t + 4 <= count) p1 = __ldcs(args.p_val + un.x + t + 4);
        const int2 un_next2 = load_unit(next + n_warps);
        const Cols8 cols_next = load_cols(next);
        float acc[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) acc[i] = 0.f;
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int q = 0; q < kPairs; ++q) {
                const bool last = q == kPairs - 1, end = last && h == 1;
                const int q_next = last ? 0 : q + 1;
                Piece a_next[2];
                load_a(a_next, (end ? un_next.y : un.y) >> 3, q_next);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float first = dot_piece(a[0], bq[i][0], acc[4 * h + i]), both = dot_piece(a[1], bq[i][1], first);
                    acc[4 * h + i] = SPECIALS && last && off ? first : both;
                    load_b(bq[i], end ? cols_next.v[i] : last ? cols.v[4 + i] : cols.v[4 * h + i], q_next);
                }
                a[0] = a_next[0];
                a[1] = a_next[1];
            }
        const float2 dot = group4_transpose_reduce(acc, t);
        if (t <= count) __stcs(args.p_val + un.x + t, step_value<STEP>(dot.x, p0, s0));
        if (t + 4 <= count) __stcs(args.p_val + un.x + t + 4, step_value<STEP>(dot.y, p1, s1));

        if (next >= n_steps) break;   // warp-uniform
        b = next;
        un = un_next;
        un_next = un_next2;
        cols = cols_next;
    }
}

// ---- bf16 storage ----------------------------------------------------------------------------------------------------
// The products of a gathered bf16 row with its A row run on mma.sync (m16n8k16, fp32 accumulators): unpacking to fp32 and
// multiplying costs two instructions per element and was what bounded this mode.  The 16 rows of the first operand are the
// gathered B rows of the 8 slots of TWO units, the 8 columns of the second operand are the A rows of the warp step's 8
// units; of the 16 x 8 products the 2 columns that belong to the two units are kept.  The order of the k elements is free
// as long as both operands use the same one, so the fragments are exactly what a lane has loaded (LB contiguous bytes of
// its row) and nothing is shuffled: lane (slot g, part t) of a step ends up with slot g of units 2t and 2t + 1.
// 37.5 M nonzeros, B in L2: K = 32 / 64 / 128 299 / 403 / 601 us, against 375 / 512 / 912 us with unpack + FMA.  (Gathered
// rows as the second operand, one unit per instruction, doubles the number of mma: 327 / 440 / 740 us.)
template <int LB>
struct Frag {
    uint32_t r[LB / 4];
};
__device__ __forceinline__ void ld_frag(Frag<32> &f, const unsigned char *p) {
    asm volatile("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(f.r[0]), "=r"(f.r[1]), "=r"(f.r[2]), "=r"(f.r[3]), "=r"(f.r[4]), "=r"(f.r[5]), "=r"(f.r[6]), "=r"(f.r[7])
                 : "l"(p));
}
__device__ __forceinline__ void ld_frag(Frag<16> &f, const unsigned char *p) {
    asm volatile("ld.global.nc.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(f.r[0]), "=r"(f.r[1]), "=r"(f.r[2]), "=r"(f.r[3]) : "l"(p));
}
// (A, as above; the 16-byte form has no such qualifier)
__device__ __forceinline__ void ld_frag_first(Frag<32> &f, const unsigned char *p) {
    asm volatile("ld.global.nc.L2::evict_first.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(f.r[0]), "=r"(f.r[1]), "=r"(f.r[2]), "=r"(f.r[3]), "=r"(f.r[4]), "=r"(f.r[5]), "=r"(f.r[6]), "=r"(f.r[7])
                 : "l"(p));
}
__device__ __forceinline__ void ld_frag_first(Frag<16> &f, const unsigned char *p) { ld_frag(f, p); }
__device__ __forceinline__ void mma_bf16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// NP pieces of 4 * LB bytes per row (the last one may be partial), R units' rows in flight per warp.  SPECIALS, as above: the lanes
// past the end of a row read zeros in place of B as well, since the tensor cores take the products of all lanes (K = 96 / 48 / 16:
// 260 / 130 / 91 us without, 269 / 138 / 96 with it).
template <int NP, int LB, int R, int MINB, int TAIL, bool COPIES>
__global__ void __launch_bounds__(kRowSegWarps * 32, MINB) sddmm_rowseg_bf16_kernel(const RowSegArgs args) {
    const int lane = threadIdx.x & 31;
    const int t = lane & 3;        // LB-byte part of a piece
    const int grp = lane >> 2;     // slot of a gathered row, unit of an A row
    const int n_steps = (args.n_units + 7) >> 3;
    const int n_warps = static_cast<int>(gridDim.x) * kRowSegWarps;
    int b = static_cast<int>(blockIdx.x) * kRowSegWarps + (threadIdx.x >> 5);
    if (b >= n_steps) return;
    const int last_unit = args.n_units - 1, last_step = n_steps - 1;
    constexpr bool SPECIALS = TAIL == kTailSpecials;
    const bool off = TAIL != kNoTail && 4 * LB * (NP - 1) + LB * t >= args.row_bytes;   // this lane's part of the last piece lies past the row
    const uint32_t stride = args.row_stride;
    const unsigned char *At = static_cast<const unsigned char *>(args.A) + LB * t;
    const unsigned char *Bt = static_cast<const unsigned char *>(args.B) + LB * t;
    const int o_last = off ? args.row_bytes - LB - LB * t : 4 * LB * (NP - 1);   // (such a lane reads the row's last LB bytes)
    const unsigned char *zero = reinterpret_cast<const unsigned char *>(g_zero_part);
    const unsigned char *Bt_last = SPECIALS && off ? zero : Bt + o_last;   // the last piece of row r of B: r * stride_last from here
    const uint32_t stride_last = SPECIALS && off ? 0u : stride;

    struct Row {
        Frag<LB> p[NP];
    };
    auto piece_offset = [&](int p) -> int { return p == NP - 1 ? o_last : 4 * LB * p; };
    auto load_b = [&](Row &f, int col) {
        const unsigned char *q = row_at(Bt, col, stride);
#pragma unroll
        for (int p = 0; p < NP; ++p) ld_frag(f.p[p], SPECIALS && p == NP - 1 ? row_at(Bt_last, col, stride_last) : q + piece_offset(p));
    };
    auto load_a = [&](Row &f, int row) {
        const unsigned char *q = row_at(At, row, stride);
#pragma unroll
        for (int p = 0; p < NP; ++p) ld_frag_first(f.p[p], p == NP - 1 && off ? zero : q + piece_offset(p));
    };
    auto load_code = [&](int step) -> int { return __ldcs(&args.units[8 * static_cast<int64_t>(min(step, last_step)) + grp].y); };
    auto load_cols = [&](int step) -> Cols8 {   // slot grp of the step's 8 units
        Cols8 c;
        const int32_t *q = args.unit_cols + 64 * static_cast<int64_t>(min(step, last_step)) + grp;
#pragma unroll
        for (int u = 0; u < 8; ++u) c.v[u] = __ldcs(q + 8 * u);
        return c;
    };

    int code_next = load_code(b + n_warps);
    Cols8 cols = load_cols(b);
    Row a, bq[R];
    load_a(a, load_code(b) >> 3);
#pragma unroll
    for (int u = 0; u < R; ++u) load_b(bq[u], cols.v[u]);

    while (true) {
        const int next = b + n_warps;
        const int4 un = __ldcs(reinterpret_cast<const int4 *>(args.units + 8 * static_cast<int64_t>(b)) + t);   // units 2t, 2t + 1
        const int c0 = 8 * b + 2 * t <= last_unit ? (un.y & 7) : -1, c1 = 8 * b + 2 * t + 1 <= last_unit ? (un.w & 7) : -1;
        const float *sv = args.s_val + 64 * static_cast<int64_t>(b) + 16 * t + grp;
        const float s0 = COPIES ? __ldcs(sv) : __ldcs(args.s_val + un.x + min(grp, un.y & 7));
        const float s1 = COPIES ? __ldcs(sv + 8) : __ldcs(args.s_val + un.z + min(grp, un.w & 7));
        const int code_next2 = load_code(next + n_warps);
        const Cols8 cols_next = load_cols(next);
        Row a_next;
        load_a(a_next, code_next >> 3);
        float r0 = 0.f, r1 = 0.f;
#pragma unroll
        for (int u = 0; u < 8; u += 2) {
            float c[4] = {0.f, 0.f, 0.f, 0.f};
            Row &x = bq[u % R], &y = bq[(u + 1) % R];
#pragma unroll
            for (int p = 0; p < NP; ++p)
#pragma unroll
                for (int k = 0; k < LB / 4; k += 2) mma_bf16(c, x.p[p].r[k], y.p[p].r[k], x.p[p].r[k + 1], y.p[p].r[k + 1], a.p[p].r[k], a.p[p].r[k + 1]);
            load_b(x, u + R < 8 ? cols.v[(u + R) & 7] : cols_next.v[(u + R) & 7]);
            load_b(y, u + 1 + R < 8 ? cols.v[(u + 1 + R) & 7] : cols_next.v[(u + 1 + R) & 7]);
            if (u == 2 * t) {   // columns 2t (slots of unit u) and 2t + 1 (slots of unit u + 1)
                r0 = c[0];
                r1 = c[3];
            }
        }
        if (grp <= c0) __stcs(args.p_val + un.x + grp, r0 * s0);
        if (grp <= c1) __stcs(args.p_val + un.z + grp, r1 * s1);

        if (next >= n_steps) break;   // warp-uniform
        b = next;
        code_next = code_next2;
        cols = cols_next;
        a = a_next;
    }
}

// ---- row groups: segments shared by NR consecutive rows with identical column lists ---------------------------------
// Block-structured matrices (several unknowns per mesh node) repeat one column list over the G rows of a block row.
// A unit of such a group covers 8 columns of the shared list for all G rows: each B row is gathered ONCE and dotted
// with G rows of A, so the traffic between L2 and the SM -- what bounds the gather -- drops by the factor G.
//   ghdr[u]  .x = CSR position of the segment in the group's first row, .y = first row * 8 + (count - 1),
//            .z = row length L (row t of the group holds the segment at .x + t * L: equal lengths, consecutive rows),
//            .w = rows that share the unit (1 for rows outside matching groups, else G)
// fp32 storage, rows of at most 8 * LPR elements, LPR in {4, 8, 16, 32}; NR = G.  A unit is taken by a group of LPR
// lanes, lane t of it holds bytes [32 t, 32 t + 32) of every row: a row of A or B is ONE 256-bit load.  36.8 M nonzeros in
// 3 x 3 blocks, K = 32 / 64: 165 / 263 us, against 206 / 292 us for rows in pieces of 16 bytes on 8 lanes (twice the load instructions,
// 64-bit index arithmetic and a shuffle per column index; 3 CTAs per SM at K = 32).
// What bounds it: the load/store unit, 139 wavefronts of 128 bytes per 32 columns at K = 64 with RUN = 2 (B rows 64, shuffles of the
// reduction 22, A rows 12 by the count of the loads, indices, S and P the rest), and the latency that 16 warps leave.  So RUN units of
// one row group go to the same lanes, one after the other, and its rows of A stay in registers from one to the next (with RUN = 1
// they are 24 wavefronts):
// RUN = 1 / 2 / 4, K = 64: 273 / 263 / 274 us, K = 32, where a row is half as long, 165 / 171 / 188; 14 M nonzeros, K = 128:
// 210 / 198 / 200, 7 M, K = 256 (two partial units of a row weigh more there): 182 / 196 / 199.  The same two by sddmm_rowseg_kernel,
// which gathers each B row three times: 423 / 409 us.
// The loads of a unit are issued together, its arithmetic and all shuffles follow.  Slower: rolling loads (a slot's registers refilled
// as soon as it is multiplied, as above) with the reduction in between 303 to 363 us; 1 / 3 CTAs per SM 344 / 316.
struct RowSegGroupArgs {
    const int4 *ghdr;          // n_units (> 0)
    const int32_t *unit_cols;  // 8 column indices per unit
    const float *s_val;        // nnz
    float *p_val;              // nnz
    const float *A;            // M rows
    const float *B;            // N rows
    int32_t n_units;
    uint32_t row_bytes;        // of a row of A or B, a multiple of 32
};

// WHOLE: a row fills its lanes.  Else (rows of 16 or 96 elements, say) the lanes past its end read its last 32 bytes once more and
// leave their products out.  20 M nonzeros, K = 8 / 16: 87 / 91 us, by sddmm_rowseg_kernel 175 / 176; 14 M, K = 96 215 (325), 7 M, K = 192 /
// 224 201 / 203 (317 / 361).  Zeros in place of both operands, from a line of their own, cost a wavefront per load: K = 96 253, K = 192 247.
template <int LPR, int NR, int RUN, bool WHOLE>
__global__ void __launch_bounds__(kRowSegWarps * 32, 2) sddmm_rowseg_group_kernel(const RowSegGroupArgs args) {
    constexpr int kRun = RUN;                    // consecutive units of a group of lanes
    constexpr int kUnits = 32 / LPR * kRun;      // per warp step
    constexpr int H = LPR == 4 ? 2 : 1;          // sums a lane ends up with (LPR > 8: its first 8 lanes)
    const int lane = threadIdx.x & 31;
    const int t = lane % LPR, grp = lane / LPR;
    const bool off = !WHOLE && 32u * t >= args.row_bytes;
    const uint32_t stride = WHOLE ? 32 * LPR : args.row_bytes, part = off ? stride - 32 : 32u * t;
    const int n_steps = (args.n_units + kUnits - 1) / kUnits;
    const int n_warps = static_cast<int>(gridDim.x) * kRowSegWarps;
    const int last_unit = args.n_units - 1;
    const unsigned char *At = reinterpret_cast<const unsigned char *>(args.A) + part;
    const unsigned char *Bt = reinterpret_cast<const unsigned char *>(args.B) + part;
    int b = static_cast<int>(blockIdx.x) * kRowSegWarps + (threadIdx.x >> 5);
    if (b >= n_steps) return;
    // unit k of this group in a warp step (k = kRun: the first one of the warp's next step)
    auto unit_index = [&](int step, int k) -> int {
        const int u = kUnits * (step + k / kRun * n_warps) + kRun * grp + k % kRun;
        return u < last_unit ? u : last_unit;
    };
    auto load_unit = [&](int u) -> int4 { return __ldcs(args.ghdr + u); };
    auto load_cols = [&](int u) -> Cols8 { return ld_cols(args.unit_cols + 8 * static_cast<int64_t>(u)); };

    int4 un = load_unit(unit_index(b, 0)), un_next = load_unit(unit_index(b, 1));
    Cols8 cols = load_cols(unit_index(b, 0));
    Piece a[NR];
    int have = -1;   // the unit header's row whose group is in `a`
    while (true) {
#pragma unroll
        for (int k = 0; k < kRun; ++k) {
            if (kRun == 1 || __any_sync(kFullMask, (un.y >> 3) != have)) {
                have = un.y >> 3;
#pragma unroll
                for (int r = 0; r < NR; ++r) a[r] = ld_piece(row_at(At, have + min(r, un.w - 1), stride));
            }
            Piece bq[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) bq[i] = ld_piece(row_at(Bt, cols.v[i], stride));
            float sv[H][NR];
#pragma unroll
            for (int h = 0; h < H; ++h)
#pragma unroll
                for (int r = 0; r < NR; ++r) sv[h][r] = __ldcs(args.s_val + un.x + min(t + 4 * h, un.y & 7) + min(r, un.w - 1) * un.z);
            const int4 un_next2 = load_unit(unit_index(b, k + 2));
            cols = load_cols(unit_index(b, k + 1));
            float acc[NR][8];
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int r = 0; r < NR; ++r) {
                    const float dot = dot_piece(a[r], bq[i], 0.f);
                    acc[r][i] = off ? 0.f : dot;
                }
            const int n = kUnits * b + kRun * grp + k <= last_unit ? (un.y & 7) : -1;
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                const bool live = r < un.w;
                float *p = args.p_val + un.x + t + r * un.z;
                if constexpr (LPR >= 8) {
                    float dot = group8_transpose_reduce(acc[r], t);
#pragma unroll
                    for (int o = 8; o < LPR; o *= 2) dot += __shfl_xor_sync(kFullMask, dot, o);
                    if (live && t <= n) __stcs(p, dot * sv[0][r]);
                } else {
                    const float2 dot = group4_transpose_reduce(acc[r], t);
                    if (live && t <= n) __stcs(p, dot.x * sv[0][r]);
                    if (live && t + 4 <= n) __stcs(p + 4, dot.y * sv[H - 1][r]);
                }
            }
            un = un_next;
            un_next = un_next2;
        }
        b += n_warps;
        if (b >= n_steps) break;   // warp-uniform
    }
}

// The same for bf16 storage, on mma.sync as sddmm_rowseg_bf16_kernel: the 16 rows of the first operand are the gathered B rows of the 8
// slots of two units, the 8 columns of the second one are the rows of A of their groups, 4 (of which NR count) for each.  Half of the
// products are used where that kernel uses an eighth, and a B row is gathered once for the group.  Lane (slot g, part t) ends up with
// slot g of the pair's unit t / 2, rows 2 (t % 2) and 2 (t % 2) + 1 of its group.  NP pieces of 4 * LB bytes per row, whole rows.
// A step is 8 units, PAIRS pairs of them at a time.  36.8 M nonzeros in 3 x 3 blocks, K = 32 / 64, by sddmm_rowseg_bf16_kernel 243 / 345 us,
// with PAIRS = 4 149 / 239, 2 188 / 210; 20 M, K = 128 (96 the same), 312, PAIRS = 2 161, 1 150; 12 M, K = 192, 285 -> 122; 10 M, K = 256
// (192 bytes spilled), 299 -> 172.
template <int NP, int LB, int PAIRS>
__global__ void __launch_bounds__(kRowSegWarps * 32, 2) sddmm_rowseg_group_bf16_kernel(const RowSegGroupArgs args) {
    constexpr uint32_t kRowBytes = 4 * LB * NP;
    const int lane = threadIdx.x & 31, t = lane & 3, grp = lane >> 2;
    const int n_steps = (args.n_units + 7) >> 3, last_unit = args.n_units - 1;
    const int n_warps = static_cast<int>(gridDim.x) * kRowSegWarps;
    const unsigned char *At = reinterpret_cast<const unsigned char *>(args.A) + LB * t;
    const unsigned char *Bt = reinterpret_cast<const unsigned char *>(args.B) + LB * t;
    int b = static_cast<int>(blockIdx.x) * kRowSegWarps + (threadIdx.x >> 5);
    if (b >= n_steps) return;

    struct Row {
        Frag<LB> p[NP];
    };
    auto load_row = [&](Row &f, const unsigned char *base, int row) {
        const unsigned char *q = row_at(base, row, kRowBytes);
#pragma unroll
        for (int p = 0; p < NP; ++p) ld_frag(f.p[p], q + 4 * LB * p);
    };
    auto load_unit = [&](int step) -> int4 { return __ldcs(args.ghdr + min(8 * step + (lane & 7), last_unit)); };   // unit lane % 8 of a step
    auto load_cols = [&](int step) -> Cols8 {   // slot grp of the step's 8 units
        Cols8 c;
#pragma unroll
        for (int u = 0; u < 8; ++u) c.v[u] = __ldcs(args.unit_cols + 8 * static_cast<int64_t>(min(8 * step + u, last_unit)) + grp);
        return c;
    };

    int4 un = load_unit(b);
    Cols8 cols = load_cols(b);
    while (true) {
        const int next = b + n_warps;
        const int4 un_next = load_unit(next);
        const Cols8 cols_next = load_cols(next);
#pragma unroll
        for (int g = 0; g < 4; g += PAIRS) {
            Row a[PAIRS], x[PAIRS], y[PAIRS];
            float s0[PAIRS], s1[PAIRS];
#pragma unroll
            for (int i = 0; i < PAIRS; ++i) {
                const int u = 2 * (g + i);
                const int ua = u + (grp >> 2);
                const int row = __shfl_sync(kFullMask, un.y, ua) >> 3, rows = __shfl_sync(kFullMask, un.w, ua);
                load_row(a[i], At, row + min(grp & 3, rows - 1));
                load_row(x[i], Bt, cols.v[u]);
                load_row(y[i], Bt, cols.v[u + 1]);
            }
            bool on0[PAIRS], on1[PAIRS];
            int at[PAIRS], step_l[PAIRS];
#pragma unroll
            for (int i = 0; i < PAIRS; ++i) {
                const int uo = 2 * (g + i) + (t >> 1), r = 2 * (t & 1);
                const int start = __shfl_sync(kFullMask, un.x, uo), code = __shfl_sync(kFullMask, un.y, uo);
                const int len = __shfl_sync(kFullMask, un.z, uo), rows = __shfl_sync(kFullMask, un.w, uo);
                const bool live = grp <= (code & 7) && 8 * b + uo <= last_unit;
                on0[i] = live && r < rows;
                on1[i] = live && r + 1 < rows;
                at[i] = start + grp + r * len;
                step_l[i] = len;
                s0[i] = on0[i] ? __ldcs(args.s_val + at[i]) : 0.f;
                s1[i] = on1[i] ? __ldcs(args.s_val + at[i] + len) : 0.f;
            }
#pragma unroll
            for (int i = 0; i < PAIRS; ++i) {
                float c[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                for (int p = 0; p < NP; ++p)
#pragma unroll
                    for (int k = 0; k < LB / 4; k += 2)
                        mma_bf16(c, x[i].p[p].r[k], y[i].p[p].r[k], x[i].p[p].r[k + 1], y[i].p[p].r[k + 1], a[i].p[p].r[k], a[i].p[p].r[k + 1]);
                const bool second = t >= 2;   // columns 4 .. 7 belong to the second unit, whose slots are rows 8 .. 15
                if (on0[i]) __stcs(args.p_val + at[i], (second ? c[2] : c[0]) * s0[i]);
                if (on1[i]) __stcs(args.p_val + at[i] + step_l[i], (second ? c[3] : c[1]) * s1[i]);
            }
        }
        if (next >= n_steps) break;   // warp-uniform
        b = next;
        un = un_next;
        cols = cols_next;
    }
}

}  // namespace sddmm
