// C-ABI implementation of the B200 SDDMM engine (see include/sddmm_b200.h).
//
// One engine = one CUDA device, one stream, one device arena that is reused
// across uploads.  upload_*() copies the operands, validates the pattern on the
// device, builds the row-length histogram and the kernel plan; run() enqueues
// the kernels (of a plan that is run often as one CUDA graph); download()
// copies P.val back.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdarg>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <new>
#include <utility>
#include <vector>

#include "../../include/sddmm_b200.h"
#include "device_pool.cuh"
#include "host_staging.cuh"
#include "kernel_dense_fma.cuh"
#include "kernel_dense_tile.cuh"
#include "kernel_rowgroup.cuh"
#include "kernel_rowseg.cuh"
#include "kernel_rowtile.cuh"
#include "kernel_spmm.cuh"
#include "plan_kernels.cuh"
#include "plan_sizes.cuh"
#include "unit_plan.cuh"

using namespace sddmm;

namespace {

constexpr size_t kAlign = 256;
constexpr int kBlock = 256;
constexpr int kMaxStageBytes = 32 * 1024;  // A rows per stage buffer (a CTA holds two)
constexpr int kTileHintShare = 64;         // fp32 mode: one nonzero in this many has to look as if it started a row of a tile
constexpr int kDenseMinCount = 2048;       // a 64x64 tile is "dense" from half full
static_assert(kTileMinOwned == kDenseMinCount / 2, "overlapping tiles stay when they own a quarter of a tile");

struct Carve {
    size_t off = 0;
    size_t take(size_t bytes) {
        const size_t o = off;
        off += (bytes + kAlign - 1) / kAlign * kAlign;
        return o;
    }
};

}  // namespace

struct sddmm_b200_engine {
    int device = 0;
    int mode = SDDMM_B200_FP32;
    uint32_t flags = 0;
    cudaStream_t stream = nullptr;
    cudaStream_t side_stream = nullptr;   // residual row-tile kernel runs here, concurrently with the dense tiles
    static constexpr int kMaxKernels = 4;
    cudaEvent_t ev_begin[kMaxKernels] = {nullptr, nullptr, nullptr, nullptr};  // per kernel, on the stream it runs on
    cudaEvent_t ev_end[kMaxKernels] = {nullptr, nullptr, nullptr, nullptr};
    cudaEvent_t ev_run0 = nullptr, ev_run1 = nullptr;   // whole run(), on the main stream (recorded once run times have been asked for)
    cudaEvent_t ev_fork = nullptr, ev_join = nullptr;
    // A held plan is replayed as a CUDA graph (built node by node, see RunTarget): measured on one kernel of 5 us, run + sync takes 7.6 us as a graph launch,
    // 12 us as a kernel launch, 14.3 us as either between two timing events and 28.7 us with the error word cleared and
    // copied back around them (what every run did before).
    cudaGraphExec_t graph = nullptr;
    static constexpr int kGraphAfter = 8;   // building one costs 90 us, replaying it saves about 12 us a run
    int runs_of_plan = 0;          // runs since the last upload (or change of a knob)
    bool run_timing = false;       // last_run_ms has been called: run() records the event pair
    bool last_run_timed_whole = false;
    // chunked host-to-host calls (pipeline.cuh): copies of consecutive row chunks are chained through these
    cudaEvent_t ev_h2d = nullptr;                 // recorded after the upload's copies are enqueued
    cudaEvent_t h2d_after = nullptr;              // another engine's ev_h2d: this upload's copies start after it
    const float *B_on_device = nullptr;           // B already in this GPU's memory (another engine's copy): taken from there
    void (*on_copies_enqueued)(void *) = nullptr; // called once ev_h2d is recorded
    void *on_copies_user = nullptr;
    int32_t coo_row_base = 0;                     // COO upload of a row slice of a larger matrix: first row of the slice
    const char *kernel_name[kMaxKernels] = {nullptr, nullptr, nullptr, nullptr};
    int kernels_launched = 0;
    bool kernel_timing = false;    // record an event pair around every kernel (sddmm_b200_set_kernel_timing)
    bool last_run_timed = false;   // ... and whether the last run() did
    int sm_count = 148;
    char err[512] = {0};

    Arena arena;
    bool uploaded = false;
    bool ran = false;
    int64_t M = 0, N = 0, K = 0, nnz = 0;

    // device views into the arena
    int32_t *d_rp = nullptr, *d_col = nullptr;
    float *d_sval = nullptr, *d_pval = nullptr;
    float *d_A32 = nullptr, *d_B32 = nullptr;
    __nv_bfloat16 *d_A16 = nullptr, *d_B16 = nullptr;
    uint32_t *d_touched = nullptr;      // one bit per column (with d_pc and d_rowstart in one piece that is cleared at once)
    size_t plan_clear_bytes = 0;
    uint32_t *d_rowstart = nullptr;
    int2 *d_item_rows = nullptr;
    int32_t *d_coo_rows = nullptr;
    PlanCounters *d_pc = nullptr;
    int32_t *h_err = nullptr;  // error word of the kernels' bounded waits, in pinned host memory (see record_error)
    int32_t *d_specials = nullptr, *h_specials = nullptr;   // set by the conversion of B: a non-finite element in the last part of a row
    bool specials = false, specials_known = false;          // ... as the host has read it back
    bool graph_specials = false;                            // ... and what the graph's kernels were chosen by
    PlanCounters *h_pc = nullptr;  // pinned landing place of the plan counters (a pageable target would make the copy a staged, blocking one)

    // dense-tile (tensor-core) path
    bool dense_possible = false;   // buffers carved for this upload
    int64_t tile_grid = 0;         // (M/64 rounded up) * (N/64 rounded up)
    int32_t tiles_per_row = 0;
    int32_t dense_cap = 0;
    bool aligned_possible = false; // the 64-grid of aligned tiles is small enough to be counted cell by cell
    int32_t *d_tile_counts = nullptr;
    int2 *d_dense_origin = nullptr;     // {first row, first column} of every dense tile (aligned detection)
    int2 *d_dense_origin2 = nullptr;    // ... (arbitrary-offset detection); `dense_origin` points at the list in use
    const int2 *dense_origin = nullptr;
    bool dense_own = false;             // the tiles in use may overlap: the kernel looks at their own masks
    int seg_slices = 1;                 // row-segment path: K is taken in this many slices of slice_cols columns, one launch each
    int slice_cols = 64;                // 64 or 128
    bool dense_fma = false;             // the tiles are computed in fp32 FMA instead of on the tensor cores
    bool dense_split3 = false;          // fp32-grade mode: operands through three slots, accumulator parked a tile at a time
    uint32_t *d_covered = nullptr;      // one bit per nonzero: owned by a dense tile
    uint32_t *d_cand = nullptr;         // one bit per nonzero: starts a half-full 64-column window of its row
    int2 *d_anchors = nullptr;          // candidate tile origins of the arbitrary-offset detection
    int32_t *d_anchor_counts = nullptr;
    int32_t anchor_cap = 0;
    DenseTileDesc *d_dense_descs = nullptr;
    int32_t *d_item_covered = nullptr;
    int32_t *d_item_ids = nullptr;
    float *d_Ax = nullptr, *d_Bx = nullptr;   // fp32_tc: [lo|hi|hi] and [hi|lo|hi] rows, 3K long
    CUtensorMap map_a, map_b;
    int32_t n_dense = 0;
    int32_t n_residual_items = 0;

    // row-group path (aligned groups of rows with one column list)
    uint8_t *d_group_ok = nullptr;
    int32_t rg_rows = 0;           // rows per group (2, 3, 4) when the row-group kernel runs, else 0
    int32_t rg_first = 0;          // first row of the first full group
    int32_t rg_groups = 0;         // ceil(M / rg_rows)

    // row-segment path (short and power-law rows; column panels when B is much larger than L2)
    int2 *d_units = nullptr;
    int32_t *d_unit_cols = nullptr;    // 8 column indices per unit
    float *d_unit_sval = nullptr;      // column panels: 8 S values per unit
    bool seg_copies = false;           // ... in use by the current plan
    int32_t *d_unit_off = nullptr;     // residual lists: per row, units before it (scan of the counts)
    int32_t *d_scan_tiles = nullptr;   // sums of the scan tiles of a list ...
    int64_t scan_cap = 0;              // ... and how many there is room for
    // Operand rows as the row-segment kernels read them: rows of Ks elements, a multiple of 32 bytes.  Ks = K where K is
    // one already (A, B themselves), else zero-padded copies.
    int64_t Ks = 0;
    float *d_Ap = nullptr, *d_Bp = nullptr;
    bool d_Ap_wanted = false;
    bool values_built = false;         // the list came with the units' copies of the S values
    bool slice_major = false;   // ... slice of K after slice of K, each of rows of slice_cols elements
    bool group_tried = false;          // a grouping was matched exactly and then dropped
    bool copies_joined = false;        // the upload's copies and conversions are already ordered before the plan's read-back
    int64_t unit_cap = 0;
    int32_t panels_plain = 1;          // column panels when every row is cut
    int32_t panels_long = 1, long_threshold = 0;   // ... when only rows of at least long_threshold (> 0) nonzeros are; the row statistics choose
    int32_t n_units = 0;
    bool use_seg = false;
    bool seg_residual = false;         // the row-segment kernel computes what the dense tiles left (units over the uncovered runs)
    int l2_bytes = 0;
    // tuning knobs (sddmm_b200_set_knob; defaults from the environment at create): < 0 = decide automatically
    double knob_panels = -1, knob_panel_mb = -1, knob_rowseg = -1, knob_group_units = -1,
           knob_offset_tiles = -1, knob_dense_split3 = -1, knob_k_slices = -1, knob_long_rows = -1;
    bool rg_units = false;             // row groups run as shared segments (row-segment group kernel) instead of the warp-per-group kernel

    HostStager stager, stager2;   // pageable host memory goes through pinned ring buffers filled by a pool of host threads (one per stream)

    // B received from another engine (sddmm_b200_stage_b): the next upload may pass B = NULL
    Arena b_stage_arena;
    float *b_stage = nullptr;
    int64_t b_stage_n = 0, b_stage_k = 0;   // dimensions of the staged B (0: none)
    cudaEvent_t ev_stage = nullptr;

    // consumer of P on the device (Y = P X): its own buffers, grown on demand, and its own plain unit list
    Arena spmm_arena;
    int32_t spmm_units = 0;            // units in the consumer's list for the current upload (0: not built yet)
    uint64_t spmm_list_in = 0;         // which buffer of spmm_arena it lies in
    int64_t spmm_k2 = 0;
    float *d_X = nullptr, *d_Y = nullptr;
    int2 *d_spmm_units = nullptr;
    cudaEvent_t ev_spmm0 = nullptr, ev_spmm1 = nullptr;
    // Y goes back to the host in up to kSpmmChunks row ranges, each as soon as its part of the kernel is done
    static constexpr int kSpmmChunks = 8;
    cudaEvent_t ev_chunk[kSpmmChunks] = {};
    int32_t spmm_cut[kSpmmChunks + 1] = {};   // units before row range c

    // plan
    sddmm_b200_plan_info plan;
    bool use_scalar = false;
    int cpl = 1;
};

namespace {

int fail(sddmm_b200_engine *e, int code, const char *fmt, ...) {
    if (e) {
        va_list ap;
        va_start(ap, fmt);
        vsnprintf(e->err, sizeof(e->err), fmt, ap);
        va_end(ap);
    }
    return code;
}

#define CU_TRY(e, call)                                                                                  \
    do {                                                                                                 \
        cudaError_t _st = (call);                                                                        \
        if (_st != cudaSuccess) {                                                                        \
            return fail((e), _st == cudaErrorMemoryAllocation ? SDDMM_B200_ERR_OOM : SDDMM_B200_ERR_CUDA, \
                        "%s failed: %s (%s:%d)", #call, cudaGetErrorString(_st), __FILE__, __LINE__);    \
        }                                                                                                \
    } while (0)

struct DeviceGuard {
    int prev = -1;
    bool ok = false, changed = false;
    explicit DeviceGuard(int dev) {
        if (cudaGetDevice(&prev) != cudaSuccess) return;
        changed = prev != dev;
        ok = !changed || cudaSetDevice(dev) == cudaSuccess;
    }
    ~DeviceGuard() {
        if (changed && prev >= 0) cudaSetDevice(prev);
    }
};

// the graph belongs to one plan: an upload, a knob or new launch arguments end it
void drop_graph(sddmm_b200_engine *e) {
    if (e->graph) cudaGraphExecDestroy(e->graph);
    e->graph = nullptr;
    e->runs_of_plan = 0;
}

int grid_for(int64_t n, int block, int cap) {
    int64_t g = (n + block - 1) / block;
    if (g < 1) g = 1;
    if (g > cap) g = cap;
    return static_cast<int>(g);
}

int grow_arena(sddmm_b200_engine *e, Arena &arena, size_t bytes, const char *what) {
    if (bytes <= arena.cap) return SDDMM_B200_OK;
    if (arena.base) {   // nothing of this engine's may still be using it
        CU_TRY(e, cudaStreamSynchronize(e->stream));
        CU_TRY(e, cudaStreamSynchronize(e->side_stream));
    }
    if (!arena.grow(e->device, bytes)) return fail(e, SDDMM_B200_ERR_OOM, "%s of %zu bytes: out of memory", what, bytes);
    return SDDMM_B200_OK;
}
int ensure_arena(sddmm_b200_engine *e, size_t bytes) { return grow_arena(e, e->arena, bytes, "device arena"); }

// Upper bound of the row-tile kernel's dynamic shared memory: two buffers of kMaxStageBytes of A rows plus a row_ptr
// slice of at most kMaxStageBytes / 16 + 1 entries (the shortest staged row is 16 bytes).
constexpr int kRowTileMaxSmem = 2 * (kMaxStageBytes + (kMaxStageBytes / 16 + 1) * 4 + 32);

// cudaFuncAttributeMaxDynamicSharedMemorySize belongs to a (function, device) pair, not to an engine: it is raised
// ONCE per pair to the upper bound, so that engines that share a GPU (chunked calls, a device listed twice, the
// allocation-free entry) can never leave each other with a limit below what their own launch asks for.
int ensure_dynamic_smem_limit(const void *fn, int device, int bytes) {
    static std::mutex mu;
    static std::map<std::pair<const void *, int>, int> raised;
    std::lock_guard<std::mutex> lock(mu);
    int &have = raised[{fn, device}];
    if (have >= bytes) return SDDMM_B200_OK;
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes) != cudaSuccess) {
        cudaGetLastError();
        return SDDMM_B200_ERR_CUDA;
    }
    have = bytes;
    return SDDMM_B200_OK;
}

template <typename ET>
using RowTileFn = void (*)(const RowTileArgs);

template <typename ET>
RowTileFn<ET> pick_rowtile(int cpl, bool exact) {
    switch (cpl) {
        case 1: return exact ? sddmm_rowtile_kernel<1, true, ET> : sddmm_rowtile_kernel<1, false, ET>;
        case 2: return exact ? sddmm_rowtile_kernel<2, true, ET> : sddmm_rowtile_kernel<2, false, ET>;
        case 4: return exact ? sddmm_rowtile_kernel<4, true, ET> : sddmm_rowtile_kernel<4, false, ET>;
        case 8: return exact ? sddmm_rowtile_kernel<8, true, ET> : sddmm_rowtile_kernel<8, false, ET>;
        default: return nullptr;
    }
}

int round_up_cpl(int64_t K) {
    const int64_t need = (K + 31) / 32;
    if (need <= 1) return 1;
    if (need <= 2) return 2;
    if (need <= 4) return 4;
    if (need <= 8) return 8;
    return 0;
}

size_t elem_bytes(const sddmm_b200_engine *e) { return e->mode == SDDMM_B200_BF16 ? 2 : 4; }

double env_double(const char *name, double fallback) {
    const char *v = std::getenv(name);
    return v ? std::atof(v) : fallback;
}

double gathered_bytes(const sddmm_b200_engine *e, int64_t cols) { return static_cast<double>(e->N) * static_cast<double>(cols) * static_cast<double>(elem_bytes(e)); }

// K = 256 from B = 5 x L2 on, rows cut into plain panels: slices of 64 that are stored one after the other, as matrices of 64 columns
// of their own; side by side in rows of 1 KB the same slices take half as long again.  The re-ordered copies are made with every
// upload of A and B, 265 us per GB of them, and a run gains about 28 us per million nonzeros, so there have to be enough nonzeros that
// a plan which runs once is no slower either.  Upload from the device and run once / a held run, us, copies against slices of 128 in
// place: 37.5 M nonzeros, A and B 1.5 GB each 6936 / 4411 against 7187 / 5450 (12.9 nonzeros per row of A and B); 9 M in 0.3 + 0.7 GB
// 1887 / 799 against 1476 / 862 (9.1), 7.8 M in 0.3 + 1.5 GB 2367 / 951 against 2043 / 1096 (4.5).  Where only the long rows are cut into
// panels the copies lose either way (power law, 18 M: 3124 / 1405 against 2593 / 1355); the row statistics decide (build_rowseg_plan).
// Knob "k_slices" = 64: wherever K is 193 .. 256.
bool slices_apart(const sddmm_b200_engine *e) {
    if (e->mode == SDDMM_B200_BF16 || !e->use_seg || e->Ks != 256) return false;
    if (e->knob_k_slices >= 0) return e->knob_k_slices == 64;
    return e->nnz >= 16 * e->M && e->nnz >= 12 * (e->M + e->N) && gathered_bytes(e, e->Ks) > 5.0 * (e->l2_bytes > 0 ? e->l2_bytes : 96.0 * (1 << 20));
}

// Large K, fp32 storage: K is taken in slices, one launch per slice over the same unit list, each adding to P.val, where that
// makes a slice of B fit L2 (or leaves column panels room) when the whole rows do not.  Measured, whole / in slices of 64, with
// B 1 / 1.3 / 1.4 / 2.7 times L2: K = 128 371 / 342, K = 192 438 / 355, K = 128 395 / 394 and 997 / 889 us; with B 0.5 times
// L2, K = 256: 725 / 751.  Slices of 128 where K allows two of them: K = 256, B 1.4 / 2.7 / 5.5 times L2, whole / 64 / 128
// columns 925 / 1232 / 798, 518 / 493 / 420, 2378 / 2157 / 1987 us, and also with B in L2 when A is streamed (731 / 777 / 684).
// Knob "k_slices": 0 = never, 1 = slices of 64 whenever K allows, 64 = the same and stored one after the other where K is 193 .. 256,
// 128 = of 128.
void choose_k_slices(sddmm_b200_engine *e) {
    if (e->slice_major) {
        e->slice_cols = 64;
        e->seg_slices = 4;
        return;
    }
    e->slice_cols = e->Ks % 128 == 0 && (e->knob_k_slices >= 128 || (e->knob_k_slices != 1 && e->knob_k_slices != 64 && e->Ks >= 256)) ? 128 : 64;
    e->seg_slices = 1;
    const int slices = static_cast<int>(e->Ks / e->slice_cols);
    if (e->K > 256) {   // rows longer than the kernels' largest instantiation (Ks is a multiple of 64)
        e->seg_slices = slices;
        return;
    }
    if (e->mode == SDDMM_B200_BF16 || e->Ks < 128 || e->Ks % 64 != 0 || e->knob_k_slices == 0) return;
    const double l2 = e->l2_bytes > 0 ? e->l2_bytes : 96.0 * (1 << 20), row = static_cast<double>(e->Ks) * 4.0;
    const bool pays = static_cast<double>(e->N) * row > 0.9 * l2 || (e->slice_cols == 128 && static_cast<double>(e->M) * row > 2.0 * l2);
    if (e->knob_k_slices < 0 && !pays) return;
    // (rows too short for panels, and none wanted for the long ones: whole rows)
    if (e->knob_k_slices < 0 && e->nnz < 16 * e->M && e->knob_long_rows == 0) return;
    e->seg_slices = slices;
}

// Column panels of the row-segment path.  B is cut into panels when it is larger than the L2 cache, so that the gathers of
// one panel hit in L2; every panel pass reads the A rows it touches again and shortens the runs a row contributes, which
// bounds the count.  Two forms; the plan takes the second where the row statistics say so (build_rowseg_plan):
//   * plain: every row is cut;
//   * long rows: only the rows of at least `long_threshold` nonzeros are cut, the shorter ones follow whole as one more entry
//     of the panel-major list.  In power-law patterns a few percent of the rows hold most of the nonzeros and the many
//     short ones would fall into runs of one or two: 20 M nonzeros, 1 M rows, K = 64 532 us plain, 396 us; 35 M, 1.5 M rows,
//     K = 32 480 / 370 us; 36 M, 2.6 M rows, K = 32 561 us without panels, 447 us.
// Knob "long_rows": 0 = never, T >= 1 = threshold T with the panels that the "panels" knob or the rule gives.
// (K = 128: where the long rows get panels the rows are taken whole, 565 us against 586 in two slices)
bool long_rows_whole(const sddmm_b200_engine *e) { return e->seg_slices > 1 && e->Ks == 128 && e->knob_k_slices < 0; }

void choose_long_rows(sddmm_b200_engine *e) {
    e->long_threshold = 0;
    e->panels_long = 1;
    if (e->knob_long_rows == 0) return;
    const double l2 = e->l2_bytes > 0 ? e->l2_bytes : 96.0 * (1 << 20);
    const double b = gathered_bytes(e, e->seg_slices > 1 && !long_rows_whole(e) ? e->slice_cols : e->Ks);
    const bool bf = e->mode == SDDMM_B200_BF16;
    // (see kPanelsFrom.)  Power law, rows of 25 on average, without / with: K = 32, B 94 / 117 / 131 MB 178 / 172, 233 / 214, 270 / 239 us,
    // rows of 10 93 / 92, 118 / 114, 134 / 127; K = 64, 117 MB 205 / 194.  bf16, where no list is built early: from L2 on, below it a
    // held run gains less than planning costs a single one (K = 64, 117 MB, rows of 25: 305 / 276, upload and run 1063 / 1250; K = 128
    // 227 / 216, 861 / 950).
    if (b <= (bf ? 1.0 : kPanelsFrom) * l2 && !(e->knob_long_rows >= 1 && e->knob_panels >= 2)) return;
    // fp32: B 333 MB, K = 32: 4 panels 407 us, 6 402 us, 8 401 us; 189 MB, 2 / 3 / 4 / 6: 300 / 287 / 286 / 286
    // bf16, whose lists are not ordered by size and whose kernel loads all slots: a short run costs as much as a full one, so fewer
    // panels and, with few of them, shorter rows too.  36 M, 2.6 M rows, K = 32, B 166 MB: 3 panels from 64 nonzeros on 348 us, 4
    // panels from 128 on 354.
    e->panels_long = e->knob_panels >= 1 ? static_cast<int>(std::min(64.0, e->knob_panels))
                                         : static_cast<int>(std::max(bf ? 2.0 : 4.0, std::min(8.0, std::ceil(b / (0.5 * l2)))));
    if (e->panels_long < 2) return;
    // (a power of two: the histogram's bins.  fp32 from 64 nonzeros on instead, 4 panels, K = 64, rows of 10: B 117 MB 106 -> 114 us,
    // 189 MB 161 -> 166; K = 32 within 1 %)
    e->long_threshold = e->knob_long_rows >= 1 ? static_cast<int>(e->knob_long_rows) : bf && e->panels_long <= 4 ? 64 : 128;
}

int choose_panels(const sddmm_b200_engine *e) {
    if (e->knob_panels >= 1 && e->knob_panels <= 64) return static_cast<int>(e->knob_panels);
    const int64_t cols = e->seg_slices > 1 ? e->slice_cols : e->Ks;
    const double b_bytes = gathered_bytes(e, cols);
    const double l2 = e->l2_bytes > 0 ? e->l2_bytes : 96.0 * (1 << 20);
    const double mean = static_cast<double>(e->nnz) / std::max<double>(1.0, static_cast<double>(e->M));
    const bool bf = e->mode == SDDMM_B200_BF16;
    // Rows too short on average.  The longer a row of B, the more a gather that misses L2 costs against a half-empty segment.  Poisson
    // rows, without / with 2 panels: K = 32, B 186 MB, mean 11 / 13 / 15: 282 / 290, 324 / 320, 368 / 353 us; K = 64, B 371 MB, mean
    // 9 / 11 / 13 / 15: 524 / 537, 619 / 607, 723 / 685, 839 / 768; K = 96, B 346 MB, mean 10 / 13: 601 / 538, 779 / 655.
    // With B between 0.85 and 1 times L2 only longer rows gain, 1 / 2 panels: K = 32, 117 MB, mean 20 / 40: 216 / 221, 403 / 368, 131 MB 258 / 238,
    // 444 / 377; K = 64, 117 MB, mean 12 / 20 / 40: 134 / 132, 205 / 190, 364 / 326; K = 128 the same; bf16 K = 128, mean 20 / 40:
    // 199 / 202, 371 / 337; slices of K, 121 MB each, mean 12 / 24 / 50: K = 128 304 / 279, 548 / 490, 873 / 659, K = 256,
    // mean 12 / 40, 290 / 268, 790 / 617.  A single run pays for the planning, so that there has to be something to gain.  Upload and
    // run, 1 / 2 panels: K = 64, mean 20, 4.0 / 9.1 M nonzeros (1.0 / 2.3 GB of gathers) 289 / 321, 476 / 485, mean 40, 18 M (4.7) 685 / 684; K = 32,
    // 8.0 / 37 M (1.0 / 4.7) 332 / 355, 918 / 982; slices, K = 128, 5.7 / 11 M 599 / 625, 877 / 818; bf16 K = 64, mean 40, 37 M
    // 1280 / 1534, a held run 501 / 461.
    if (b_bytes <= kPanelsFrom * l2) return 1;
    if (b_bytes <= l2) {
        if (bf) return cols <= 64 || mean < 28.0 ? 1 : 2;
        if (e->seg_slices > 1) return mean < 11.0 ? 1 : 2;
        return mean < (cols <= 32 ? 24.0 : 16.0) || static_cast<double>(e->nnz) * static_cast<double>(cols) * 4.0 < 1.4e9 ? 1 : 2;
    }
    // (bf16 rows of 33 to 64, where no list is built early: a held run / upload and run, 1 / 2 panels, B 157 MB, mean 26 / 45 499 / 479, 1370 / 1597 and
    // 574 / 511, 1374 / 1579; 186 MB, mean 26 / 35 / 45 625 / 601, 1628 / 1884, 709 / 567, 1648 / 1736 and 772 / 547, 1632 / 1617; 211 MB, mean
    // 26 / 35 686 / 621, 1760 / 1971 and 823 / 591, 1837 / 1827)
    if (bf && cols > 32 && cols <= 64 && b_bytes <= (mean < 32.0 ? 1.5 : 1.3) * l2) return 1;
    // (K = 32, B 262 / 388 MB, mean 8 / 10 / 12: 347 / 342, 418 / 392, 500 / 438 and 616 / 569, 726 / 654, 719 / 638)
    if (mean < (bf ? (cols <= 32 ? 26.0 : cols <= 64 ? 20.0 : 13.0) : cols <= 32 ? (b_bytes > 1.8 * l2 ? 10.0 : 13.0) : cols <= 64 ? 11.0 : 9.0)) return 1;
    // Slices of 128 columns: panels that fit L2 one by one, if an average row has 3 nonzeros for each, or none.  Sustained, B 205 MB,
    // mean 10, 1 / 2 panels: 577 / 527 us; 358 MB, 9.6, 1 / 2 / 3: 1158 / 1174 / 1122; 461 MB, 9.5: 1549 / 1659 / 1640, 12, 1 / 2 / 3 / 4:
    // 2006 / 1999 / 1905 / 1859; longer rows, 358 MB, 30, 3 / 4 / 5: 2390 / 2086 / 2084; 512 MB, 20, 4 / 5 / 6: 2836 / 2651 / 2834; 744 MB,
    // 26, 4 / 5 / 6 / 7: 6027 / 5815 / 5538 / 5347; 210 MB, 40, 2 / 4: 828 / 711.
    if (cols == 128 && e->seg_slices > 1 && !bf) {
        const double need = std::ceil(b_bytes / l2);
        if (mean < 16.0) return 3.0 * need > mean || need > 4.0 ? 1 : static_cast<int>(need);
        return static_cast<int>(std::min(8.0, std::min(std::ceil(b_bytes / (0.6 * l2)), std::floor(mean / 3.5))));
    }
    // bf16 storage, 1 / 2 / 3 / 4 panels.  K = 64: B 157 MB, mean 14 308 / 308 / 349 / 417, 26 431 / 404 / 414 / 434, 45 414 / 377 / 372 / 386;
    // 262 MB, 26 630 / 473 / 484 / 488, 45 633 / 434 / 436 / 436.  K = 128: 157 MB, 14 230 / 215 / 265 / 294, 26 393 / 368 / 358 / 352, 45
    // 625 / 526 / 498 / 534; 388 MB, 14 908 / 725 / 749 / 831, 26 1175 / 804 / 763 / 739, 45 1521 / 764 / 679 / 652
    if (bf) {
        if (cols <= 64) return static_cast<int>(std::max(2.0, std::min(4.0, std::ceil(b_bytes / (1.25 * l2)))));
        return static_cast<int>(std::min(std::min(4.0, std::ceil(b_bytes / (0.8 * l2))), std::max(2.0, std::floor(mean / 6.0))));
    }
    // measured on B200 (126 MB of L2): a run shorter than a segment wastes gather slots, so panels of about 100 MB for rows of one
    // piece (B 199 MB, mean 26: 2 / 3 panels 344 / 365 us), 80 MB for longer rows, where a slot's waste weighs less against its row
    // (K = 64, B 179 MB: 428 / 414 us, B 372 MB: 3 / 4 panels 1138 / 1116); at most 2, or one per 6 nonzeros of an average row,
    // and never more than 4 (5: 3 % slower)
    const double panel = e->knob_panel_mb > 0 ? e->knob_panel_mb * (1 << 20) : (cols <= 32 ? 0.8 : 0.6) * l2;
    return static_cast<int>(std::min(std::ceil(b_bytes / panel), std::min(4.0, std::max(2.0, std::floor(mean / 6.0)))));
}

// Which inputs the row-segment kernels take (the scalar and the row-tile kernel are left with the rest): K below 8 that is
// no multiple of 4 stays with the scalar kernel, a padded row would be several times the real one.
bool seg_possible(const sddmm_b200_engine *e) {
    if ((e->flags & SDDMM_B200_FLAG_NO_ROW_SEGMENTS) || e->knob_rowseg == 0 || e->M >= kUnitRowLimit) return false;
    return e->K % 4 == 0 || e->K >= 8;
}

// How much an upload may take: what is fastest, no copies of A and B beside them, no lists (the A-row-tile and the scalar kernel
// run on the arrays as they are).  The next one is tried when the device has no room.
enum Footprint : int { kFull, kNoCopies, kNoLists };

// slices of K, column panels and the threshold of long rows, in the order in which they depend on one another
void choose_list_forms(sddmm_b200_engine *e) {
    choose_k_slices(e);
    choose_long_rows(e);
    e->panels_plain = choose_panels(e);
}

// Lay out the arena for the current dimensions and point the views into it.
int carve_arena(sddmm_b200_engine *e, bool coo, int n_items, Footprint footprint) {
    Carve c;
    const bool bf = e->mode == SDDMM_B200_BF16;
    const int64_t row = bf || footprint == kFull ? padded_row(bf, e->K) : unpadded_row(e->K);   // (bf16 rows are a copy in any case)
    e->use_seg = footprint != kNoLists && row > 0 && seg_possible(e);
    e->Ks = e->use_seg ? row : e->K;
    const size_t nnz = static_cast<size_t>(e->nnz), M = static_cast<size_t>(e->M), N = static_cast<size_t>(e->N),
                 K = static_cast<size_t>(e->K);
    const size_t o_rp = c.take((M + 1) * 4);
    const size_t o_col = c.take(nnz * 4 + 16);
    const size_t o_sv = c.take(nnz * 4 + 16);
    const size_t o_pv = c.take(nnz * 4 + 16);
    const size_t o_A = c.take(M * K * 4);
    const size_t o_B = c.take(N * K * 4);
    const size_t Ks = static_cast<size_t>(e->Ks);
    const size_t o_A16 = bf ? c.take(M * Ks * 2) : 0;
    const size_t o_B16 = bf ? c.take(N * Ks * 2) : 0;
    e->slice_major = footprint == kFull && slices_apart(e);
    const bool padded = !bf && e->use_seg && (e->Ks != e->K || e->slice_major);
    e->d_Ap_wanted = padded;
    const size_t o_Ap = padded ? c.take(M * Ks * 4) : 0;
    const size_t o_Bp = padded ? c.take(N * Ks * 4) : 0;
    const size_t o_pc = c.take(sizeof(PlanCounters));
    const size_t o_spec = c.take(sizeof(int32_t));
    const size_t o_touch = c.take((N / 32 + 1) * 4);
    const size_t o_rs = c.take((nnz / 32 + 2) * 4);
    e->plan_clear_bytes = c.off - o_pc;
    const size_t o_items = c.take(static_cast<size_t>(std::max(n_items, 1)) * sizeof(int2));
    const size_t o_coo = coo ? c.take(nnz * 4 + 16) : 0;
    const size_t o_gok = c.take(M / 2 + 4);   // one byte per row group (groups of >= 2 rows, plus the leading partial group)
    // row-segment path: unit list (upper bound: one unit per 8 nonzeros plus one ragged unit per row and panel), scan scratch
    bool any_panels = false;
    e->unit_cap = e->scan_cap = 0;
    auto room_for_lists = [&]() {
        choose_list_forms(e);
        size_t runs = std::min(M * static_cast<size_t>(e->panels_plain), nnz);
        if (e->long_threshold > 0) {   // a run per short row, and per panel for at most nnz / long_threshold long rows
            runs = std::max(runs, std::min(M + std::min(nnz / static_cast<size_t>(e->long_threshold), M) * static_cast<size_t>(e->panels_long), nnz));
        }
        any_panels = any_panels || e->panels_plain > 1 || e->long_threshold > 0;
        e->unit_cap = std::max(e->unit_cap, unit_capacity(e->nnz, static_cast<int64_t>(runs)));
        e->scan_cap = std::max(e->scan_cap, plan_tile_sums(e->M, e->panels_plain, e->long_threshold > 0 ? e->panels_long : 0));
    };
    if (e->slice_major) {   // (the row statistics may yet choose slices in place)
        e->slice_major = false;
        room_for_lists();
        e->slice_major = true;
    }
    room_for_lists();
    const size_t o_units = e->use_seg ? c.take(static_cast<size_t>(e->unit_cap + 8) * sizeof(int4)) : 0;   // (row groups use 16-byte headers)
    const size_t o_ucols = e->use_seg ? c.take(static_cast<size_t>(e->unit_cap + 8) * 32) : 0;
    const size_t o_uval = e->use_seg && any_panels ? c.take(static_cast<size_t>(e->unit_cap + 8) * 32) : 0;
    const size_t o_uoff = c.take((M + 1) * 4);
    const size_t o_stile = c.take(static_cast<size_t>(e->scan_cap) * 4);
    // dense-tile path: only carved when the mode, K and the size of the 64x64 tile grid allow it
    e->tiles_per_row = static_cast<int32_t>((N + 63) / 64);
    e->tile_grid = static_cast<int64_t>((M + 63) / 64) * e->tiles_per_row;
    // tensor-core modes.  bf16 takes the same kind::tf32 kernel: the fp32 copies of A and B are rounded to bf16 in place at
    // upload, every bf16 value is exactly a tf32 value (8 against 11 significand bits), so the tile products are exactly the
    // bf16-input / fp32-accumulate ones.
    const bool tc_mode = e->mode == SDDMM_B200_TF32 || e->mode == SDDMM_B200_FP32_TC || e->mode == SDDMM_B200_BF16;
    // fp32 mode: the same tiles in plain fp32 arithmetic (unless the row-segment path is asked for or switched off)
    const bool fma_mode = e->mode == SDDMM_B200_FP32 && e->use_seg && e->knob_rowseg != 1;
    e->dense_possible = (tc_mode || fma_mode) && !(e->flags & SDDMM_B200_FLAG_NO_DENSE_TILES) && K % 32 == 0 && K <= 256 && nnz >= kDenseMinCount;
    e->aligned_possible = e->dense_possible && e->tile_grid <= (int64_t(1) << 22);
    // (tiles at arbitrary offsets may overlap, so there can be more of them than nnz / 2048; what does not fit is dropped)
    e->dense_cap = e->dense_possible ? static_cast<int32_t>(2 * (e->nnz / kDenseMinCount) + 16) : 0;
    e->anchor_cap = e->dense_possible ? static_cast<int32_t>(e->nnz / 256 + 64) : 0;
    const bool split = e->dense_possible && e->mode == SDDMM_B200_FP32_TC;
    const size_t tg = static_cast<size_t>(e->tile_grid);
    const size_t o_tc = e->aligned_possible ? c.take(tg * 4) : 0;
    const size_t o_di = e->dense_possible ? c.take(static_cast<size_t>(e->dense_cap) * sizeof(int2)) : 0;
    const size_t o_di2 = e->dense_possible ? c.take(static_cast<size_t>(e->dense_cap) * sizeof(int2)) : 0;
    const size_t o_cov = e->dense_possible ? c.take((nnz / 32 + 2) * 4) : 0;
    const size_t o_cand = e->dense_possible ? c.take((nnz / 32 + 2) * 4) : 0;
    const size_t o_anc = e->dense_possible ? c.take(static_cast<size_t>(e->anchor_cap) * sizeof(int2)) : 0;
    const size_t o_ancc = e->dense_possible ? c.take(static_cast<size_t>(e->anchor_cap) * 4) : 0;
    const size_t o_dd = e->dense_possible ? c.take(static_cast<size_t>(e->dense_cap) * sizeof(DenseTileDesc)) : 0;
    const size_t o_ic = e->dense_possible ? c.take(static_cast<size_t>(std::max(n_items, 1)) * 4) : 0;
    const size_t o_ii = e->dense_possible ? c.take(static_cast<size_t>(std::max(n_items, 1)) * 4) : 0;
    const size_t o_ax = split ? c.take(M * K * 12) : 0;
    const size_t o_bx = split ? c.take(N * K * 12) : 0;
    int st = ensure_arena(e, c.off);
    if (st) return st;
    char *b = e->arena.base;
    e->d_tile_counts = e->aligned_possible ? reinterpret_cast<int32_t *>(b + o_tc) : nullptr;
    e->d_dense_origin = e->dense_possible ? reinterpret_cast<int2 *>(b + o_di) : nullptr;
    e->d_dense_origin2 = e->dense_possible ? reinterpret_cast<int2 *>(b + o_di2) : nullptr;
    e->d_covered = e->dense_possible ? reinterpret_cast<uint32_t *>(b + o_cov) : nullptr;
    e->d_cand = e->dense_possible ? reinterpret_cast<uint32_t *>(b + o_cand) : nullptr;
    e->d_anchors = e->dense_possible ? reinterpret_cast<int2 *>(b + o_anc) : nullptr;
    e->d_anchor_counts = e->dense_possible ? reinterpret_cast<int32_t *>(b + o_ancc) : nullptr;
    e->d_dense_descs = e->dense_possible ? reinterpret_cast<DenseTileDesc *>(b + o_dd) : nullptr;
    e->d_item_covered = e->dense_possible ? reinterpret_cast<int32_t *>(b + o_ic) : nullptr;
    e->d_item_ids = e->dense_possible ? reinterpret_cast<int32_t *>(b + o_ii) : nullptr;
    e->d_Ax = split ? reinterpret_cast<float *>(b + o_ax) : nullptr;
    e->d_Bx = split ? reinterpret_cast<float *>(b + o_bx) : nullptr;
    e->d_units = e->use_seg ? reinterpret_cast<int2 *>(b + o_units) : nullptr;
    e->d_unit_cols = e->use_seg ? reinterpret_cast<int32_t *>(b + o_ucols) : nullptr;
    e->d_unit_sval = e->use_seg && any_panels ? reinterpret_cast<float *>(b + o_uval) : nullptr;
    e->d_Ap = padded ? reinterpret_cast<float *>(b + o_Ap) : nullptr;
    e->d_Bp = padded ? reinterpret_cast<float *>(b + o_Bp) : nullptr;
    e->d_unit_off = reinterpret_cast<int32_t *>(b + o_uoff);
    e->d_scan_tiles = reinterpret_cast<int32_t *>(b + o_stile);
    e->d_rp = reinterpret_cast<int32_t *>(b + o_rp);
    e->d_group_ok = reinterpret_cast<uint8_t *>(b + o_gok);
    e->d_col = reinterpret_cast<int32_t *>(b + o_col);
    e->d_sval = reinterpret_cast<float *>(b + o_sv);
    e->d_pval = reinterpret_cast<float *>(b + o_pv);
    e->d_A32 = reinterpret_cast<float *>(b + o_A);
    e->d_B32 = reinterpret_cast<float *>(b + o_B);
    e->d_A16 = bf ? reinterpret_cast<__nv_bfloat16 *>(b + o_A16) : nullptr;
    e->d_B16 = bf ? reinterpret_cast<__nv_bfloat16 *>(b + o_B16) : nullptr;
    e->d_touched = reinterpret_cast<uint32_t *>(b + o_touch);
    e->d_rowstart = reinterpret_cast<uint32_t *>(b + o_rs);
    e->d_item_rows = reinterpret_cast<int2 *>(b + o_items);
    e->d_coo_rows = coo ? reinterpret_cast<int32_t *>(b + o_coo) : nullptr;
    e->d_pc = reinterpret_cast<PlanCounters *>(b + o_pc);
    e->d_specials = reinterpret_cast<int32_t *>(b + o_spec);
    return SDDMM_B200_OK;
}

// Work-item size: 2048 nonzeros, smaller for small matrices so that every SM gets work.
int choose_item_nnz(const sddmm_b200_engine *e) {
    if (const char *env = std::getenv("SDDMM_B200_ITEM_NNZ")) {  // tuning knob: nonzeros per work item
        const long v = std::atol(env);
        if (v >= 32 && v <= (1 << 20)) return static_cast<int>((v + 31) / 32 * 32);
    }
    const int64_t per = e->nnz / (static_cast<int64_t>(e->sm_count) * 4);
    int64_t z = (per + 31) / 32 * 32;
    z = std::max<int64_t>(256, std::min<int64_t>(2048, z));
    return static_cast<int>(z);
}

// bytes of a row that hold elements, in whole 32-byte parts (bf16 rows of at most 32 elements: 16-byte parts)
int32_t seg_part_bytes(const sddmm_b200_engine *e) { return e->mode == SDDMM_B200_BF16 && e->Ks <= 32 ? 16 : 32; }
int32_t seg_row_bytes(const sddmm_b200_engine *e) {
    const int64_t bytes = e->K * static_cast<int64_t>(elem_bytes(e)), part = seg_part_bytes(e);
    return static_cast<int32_t>((bytes + part - 1) / part * part);
}
// rows whose last piece is partial: some lanes of the row-segment kernels lie past their end (not in slices of K, which are whole)
bool ragged_rows(const sddmm_b200_engine *e) { return e->use_seg && e->K <= 256 && seg_row_bytes(e) % (4 * seg_part_bytes(e)) != 0; }
// ... and whether they have to leave the product out (see SPECIALS in kernel_rowseg.cuh): always in fp32 rows of one piece, else
// where the last conversion of B has seen a non-finite element in a row's last part, where it is still under way, and where there
// is none because the kernel reads B itself
bool leave_out_past_end(const sddmm_b200_engine *e) {
    if (!ragged_rows(e) || e->seg_slices > 1) return false;
    if (e->mode != SDDMM_B200_BF16 && (e->Ks <= 32 || !e->d_Bp)) return true;
    return !e->specials_known || e->specials;
}
// Once the stream has drained after convert_storage: what it has seen.
void settle_specials(sddmm_b200_engine *e) {
    e->specials = *static_cast<volatile int32_t *>(e->h_specials) != 0;
    e->specials_known = true;
}

// the units' copies of S.val follow every change of S.val
int refresh_unit_values(sddmm_b200_engine *e) {
    if (!e->use_seg || !e->seg_copies || e->n_units == 0) return SDDMM_B200_OK;
    k_unit_values<<<grid_for(8 * static_cast<int64_t>(e->n_units), kBlock, e->sm_count * 32), kBlock, 0, e->stream>>>(e->d_units, e->n_units, e->d_sval,
                                                                                                                e->d_unit_sval);
    CU_TRY(e, cudaGetLastError());
    return SDDMM_B200_OK;
}

int convert_storage(sddmm_b200_engine *e) {
    const int cap = e->sm_count * 8;
    e->specials_known = false;
    int32_t *const seen = ragged_rows(e) ? e->d_specials : nullptr;
    const int32_t last_part = static_cast<int32_t>((seg_row_bytes(e) - seg_part_bytes(e)) / static_cast<int32_t>(elem_bytes(e)));
    *static_cast<volatile int32_t *>(e->h_specials) = 0;
    if (seen) CU_TRY(e, cudaMemsetAsync(seen, 0, sizeof(int32_t), e->stream));
    if (int rc = refresh_unit_values(e)) return rc;
    if (e->d_Ax && e->n_dense > 0) {  // hi/lo-concatenated operands of the fp32-grade tensor-core mode (only when tiles were found)
        k_split_concat_tf32<<<grid_for(e->M * e->K, kBlock, cap), kBlock, 0, e->stream>>>(e->d_A32, e->d_Ax, e->M, static_cast<int32_t>(e->K), 1);
        k_split_concat_tf32<<<grid_for(e->N * e->K, kBlock, cap), kBlock, 0, e->stream>>>(e->d_B32, e->d_Bx, e->N, static_cast<int32_t>(e->K), 0);
        CU_TRY(e, cudaGetLastError());
    }
    const int32_t K = static_cast<int32_t>(e->K), Ks = static_cast<int32_t>(e->Ks);
    if (e->d_Ap) {
        k_pad_rows<<<grid_for(e->M * (Ks / 4), kBlock, cap), kBlock, 0, e->stream>>>(e->d_A32, e->d_Ap, e->M, K, Ks, e->slice_major ? e->slice_cols : Ks, 0, nullptr);
        k_pad_rows<<<grid_for(e->N * (Ks / 4), kBlock, cap), kBlock, 0, e->stream>>>(e->d_B32, e->d_Bp, e->N, K, Ks, e->slice_major ? e->slice_cols : Ks, last_part, seen);
        CU_TRY(e, cudaGetLastError());
    }
    if (e->mode == SDDMM_B200_BF16) {   // (the fp32 copies keep the rounded values: the dense-tile kernel reads them through its tensor maps)
        k_f32_to_bf16<<<grid_for(e->M * (Ks / 4), kBlock, cap), kBlock, 0, e->stream>>>(e->d_A32, e->d_A16, e->M, K, Ks, 0, nullptr);
        k_f32_to_bf16<<<grid_for(e->N * (Ks / 4), kBlock, cap), kBlock, 0, e->stream>>>(e->d_B32, e->d_B16, e->N, K, Ks, last_part, seen);
        CU_TRY(e, cudaGetLastError());
    }
    if (seen) CU_TRY(e, cudaMemcpyAsync(e->h_specials, seen, sizeof(int32_t), cudaMemcpyDeviceToHost, e->stream));
    return SDDMM_B200_OK;
}

// 2-D tensor map over a row-major rows x K fp32 matrix: box = 32 floats (one 128-byte
// k-block) x 64 rows, 128-byte swizzle, out-of-range rows read as zero.
int make_operand_map(sddmm_b200_engine *e, CUtensorMap *map, const float *base, int64_t rows, int64_t K) {
    typedef CUresult (*EncodeFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                                 const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                                 CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static EncodeFn encode = nullptr;
    if (!encode) {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult qres;
        CU_TRY(e, cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &qres));
        if (!fn || qres != cudaDriverEntryPointSuccess) return fail(e, SDDMM_B200_ERR_CUDA, "cuTensorMapEncodeTiled not available");
        encode = reinterpret_cast<EncodeFn>(fn);
    }
    const cuuint64_t gdim[2] = {static_cast<cuuint64_t>(K), static_cast<cuuint64_t>(rows)};
    const cuuint64_t gstride[1] = {static_cast<cuuint64_t>(K) * 4};
    const cuuint32_t box[2] = {32, 64};
    const cuuint32_t estride[2] = {1, 1};
    const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float *>(base), gdim, gstride, box, estride,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(e, SDDMM_B200_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", static_cast<int>(r));
    return SDDMM_B200_OK;
}

// Find the 64x64 tiles that are at least half full, build their row descriptors and the list
// of work items the row-tile kernel still has to visit.
// the plan counters as they are when the stream has drained
int read_counters(sddmm_b200_engine *e, PlanCounters *out) {
    CU_TRY(e, cudaMemcpyAsync(e->h_pc, e->d_pc, sizeof(PlanCounters), cudaMemcpyDeviceToHost, e->stream));
    CU_TRY(e, cudaStreamSynchronize(e->stream));
    *out = *e->h_pc;
    return SDDMM_B200_OK;
}

int cuda_status(sddmm_b200_engine *e, cudaError_t err);

// Before a scan is launched: the memory laid out for its tile sums has to hold them.
int check_tile_sums(sddmm_b200_engine *e, int64_t tiles) {
    if (tiles <= e->scan_cap) return SDDMM_B200_OK;
    return fail(e, SDDMM_B200_ERR_CUDA, "unit list of %lld scan tiles, laid out for %lld", (long long)tiles, (long long)e->scan_cap);
}

// the instantiation of the dense-tile kernel for (own masks looked at, three-slot operand scheme)
const void *dense_function(bool own, bool split3) {
    if (split3) return own ? reinterpret_cast<const void *>(sddmm_dense_tile_kernel<true, true>) : reinterpret_cast<const void *>(sddmm_dense_tile_kernel<false, true>);
    return own ? reinterpret_cast<const void *>(sddmm_dense_tile_kernel<true, false>) : reinterpret_cast<const void *>(sddmm_dense_tile_kernel<false, false>);
}

using DenseFmaFn = void (*)(const DenseFmaArgs);
DenseFmaFn dense_fma_function(bool own) { return own ? sddmm_dense_tile_fma_kernel<true> : sddmm_dense_tile_fma_kernel<false>; }

int build_dense_plan(sddmm_b200_engine *e, const PlanCounters &base_pc, int item_nnz, int n_items) {
    e->n_dense = 0;
    e->n_residual_items = n_items;
    if (!e->dense_possible || base_pc.unsorted_cols || base_pc.dup_cols || base_pc.max_row_nnz < 32) return SDDMM_B200_OK;
    // Looking for tiles takes several passes over the pattern, so a cheap look comes first, in two steps: the column scan has
    // counted the nonzeros that start a half-full 64-column window of their row (none of every fourth one: no tile), then
    // sampled windows are compared with the rows 32 above and below.  The tensor-core modes take any tile that shows; the
    // fp32 mode, whose tiles gain less, wants about a tenth of the nonzeros in them (a quarter of a block's start a window).
    const bool fp32 = e->mode == SDDMM_B200_FP32;
    if (e->knob_offset_tiles <= 0) {
        if (base_pc.window_hint == 0 || (fp32 && base_pc.window_hint * kTileHintShare < static_cast<unsigned long long>(e->nnz))) return SDDMM_B200_OK;
        const int samples = static_cast<int>(std::min<int64_t>(e->nnz, 16384));
        k_block_sample<<<grid_for(samples, kBlock, 1 << 30), kBlock, 0, e->stream>>>(e->d_rp, e->d_col, static_cast<int32_t>(e->M), e->nnz, 32, samples, e->d_pc);
        CU_TRY(e, cudaGetLastError());
        PlanCounters seen;
        if (int rc = read_counters(e, &seen)) return rc;
        if (seen.block_samples == 0 || (fp32 && static_cast<int64_t>(seen.block_samples) * kTileHintShare < samples)) return SDDMM_B200_OK;
    }
    const int cap = e->sm_count * 8;
    cudaStream_t s = e->stream;
    const int32_t M = static_cast<int32_t>(e->M);
    CU_TRY(e, cudaMemsetAsync(e->d_covered, 0, (static_cast<size_t>(e->nnz) / 32 + 2) * 4, s));
    CU_TRY(e, cudaMemsetAsync(e->d_item_covered, 0, static_cast<size_t>(n_items) * 4, s));
    PlanCounters pc;
    // ---- tiles on the 64-grid: count every cell, keep those at least half full ----
    int n_aligned = 0;
    unsigned long long aligned_nnz = 0;
    if (e->aligned_possible) {
        CU_TRY(e, cudaMemsetAsync(e->d_tile_counts, 0, static_cast<size_t>(e->tile_grid) * 4, s));
        k_tile_count<<<grid_for(e->M * 32, kBlock, 1 << 30), kBlock, 0, s>>>(e->d_rp, e->d_col, M, e->tiles_per_row, e->d_tile_counts);
        k_tile_select<<<grid_for(e->tile_grid, kBlock, cap), kBlock, 0, s>>>(e->d_tile_counts, e->tile_grid, e->tiles_per_row, kDenseMinCount,
                                                                             e->d_dense_origin, e->dense_cap, e->d_pc);
        CU_TRY(e, cudaGetLastError());
        if (int rc = read_counters(e, &pc)) return rc;
        n_aligned = std::min(pc.dense_tiles, e->dense_cap);
        aligned_nnz = pc.window_nnz;
    }
    int n_dense = n_aligned;
    e->dense_origin = e->d_dense_origin;
    bool offsets_used = false;   // the tiles in use come from the arbitrary-offset detection (they may overlap)
    // ---- tiles at arbitrary offsets ("randomly placed blocks"): when the grid catches less than half of the nonzeros and
    //      the rows are long enough to hold half-full 64-column windows at all ----
    const bool try_offsets = e->knob_offset_tiles != 0 &&
                             (e->knob_offset_tiles > 0 || (2 * aligned_nnz < static_cast<unsigned long long>(e->nnz) &&
                                                           e->nnz >= 16 * static_cast<int64_t>(std::max<unsigned long long>(1, base_pc.rows_nonempty))));
    if (try_offsets) {
        const int wcap = e->sm_count * 32;
        CU_TRY(e, cudaMemsetAsync(e->d_cand, 0, (static_cast<size_t>(e->nnz) / 32 + 2) * 4, s));
        CU_TRY(e, cudaMemsetAsync(&e->d_pc->n_anchors, 0, sizeof(int), s));
        k_window_candidates<<<grid_for(e->M * 32, kBlock, wcap), kBlock, 0, s>>>(e->d_rp, e->d_col, M, 32, e->d_cand);
        k_window_anchors<<<grid_for(e->M * 32, kBlock, wcap), kBlock, 0, s>>>(e->d_rp, e->d_col, M, 32, e->d_cand, e->d_anchors, e->anchor_cap,
                                                                              &e->d_pc->n_anchors);
        CU_TRY(e, cudaGetLastError());
        if (int rc = read_counters(e, &pc)) return rc;
        const int n_anchors = std::min(pc.n_anchors, e->anchor_cap);
        if (n_anchors > 0) {
            CU_TRY(e, cudaMemsetAsync(e->d_anchor_counts, 0, static_cast<size_t>(n_anchors) * 4, s));
            CU_TRY(e, cudaMemsetAsync(&e->d_pc->dense_tiles, 0, sizeof(int), s));
            CU_TRY(e, cudaMemsetAsync(&e->d_pc->window_nnz, 0, sizeof(unsigned long long), s));
            k_anchor_counts<<<grid_for(static_cast<int64_t>(n_anchors) * 64, kBlock, 1 << 30), kBlock, 0, s>>>(e->d_rp, e->d_col, M, e->d_anchors,
                                                                                                            n_anchors, e->d_anchor_counts);
            k_anchor_select<<<grid_for(n_anchors, kBlock, 1 << 30), kBlock, 0, s>>>(e->d_anchors, e->d_anchor_counts, n_anchors, kDenseMinCount,
                                                                                    e->d_dense_origin2, e->dense_cap, e->d_pc);
            CU_TRY(e, cudaGetLastError());
            if (int rc = read_counters(e, &pc)) return rc;
            // (windows may overlap, so their sum can count a nonzero twice; it still ranks the two detections)
            if (pc.window_nnz > aligned_nnz) {
                n_dense = std::min(pc.dense_tiles, e->dense_cap);
                e->dense_origin = e->d_dense_origin2;
                offsets_used = true;
            }
        }
    }
    if (n_dense <= 0) return SDDMM_B200_OK;
    // row descriptors and ownership (tile_owned: the anchor counters are free again)
    auto describe = [&]() -> int {
        CU_TRY(e, cudaMemsetAsync(&e->d_pc->dense_nnz, 0, sizeof(unsigned long long), s));
        CU_TRY(e, cudaMemsetAsync(e->d_anchor_counts, 0, static_cast<size_t>(n_dense) * 4, s));
        // overlapping tiles: one owner key per nonzero, kept in P.val's storage (unused until the first run)
        uint32_t *owner = offsets_used ? reinterpret_cast<uint32_t *>(e->d_pval) : nullptr;
        if (owner) {
            CU_TRY(e, cudaMemsetAsync(owner, 0xFF, static_cast<size_t>(e->nnz) * 4, s));
            k_tile_propose<<<grid_for(static_cast<int64_t>(n_dense) * 64 * 32, kBlock, 1 << 30), kBlock, 0, s>>>(e->d_rp, e->d_col, M, e->dense_origin,
                                                                                                             n_dense, owner);
        }
        k_tile_rows<DenseTileDesc><<<grid_for(static_cast<int64_t>(n_dense) * 64 * 32, kBlock, 1 << 30), kBlock, 0, s>>>(
            e->d_rp, e->d_col, M, e->dense_origin, n_dense, e->d_dense_descs, e->d_covered, item_nnz, e->d_item_covered, e->d_anchor_counts,
            e->d_pc, owner);
        return cuda_status(e, cudaGetLastError());
    };
    if (int rc = describe()) return rc;
    if (offsets_used) {
        // windows at arbitrary offsets overlap: drop the tiles that own less than a quarter of a tile, then decide the
        // ownership afresh among those that stay
        int2 *kept = e->d_dense_origin;   // (the grid's list is not used)
        CU_TRY(e, cudaMemsetAsync(&e->d_pc->dense_tiles, 0, sizeof(int), s));
        k_tile_keep<<<grid_for(n_dense, kBlock, 1 << 30), kBlock, 0, s>>>(e->dense_origin, e->d_anchor_counts, n_dense, kTileMinOwned, kept, e->d_pc);
        CU_TRY(e, cudaGetLastError());
        if (int rc = read_counters(e, &pc)) return rc;
        if (pc.dense_tiles < n_dense) {
            n_dense = pc.dense_tiles;
            e->dense_origin = kept;
            CU_TRY(e, cudaMemsetAsync(e->d_covered, 0, (static_cast<size_t>(e->nnz) / 32 + 2) * 4, s));
            CU_TRY(e, cudaMemsetAsync(e->d_item_covered, 0, static_cast<size_t>(n_items) * 4, s));
            if (n_dense <= 0) return SDDMM_B200_OK;
            if (int rc = describe()) return rc;
        }
    }
    k_residual_items<<<grid_for(n_items, kBlock, 1 << 30), kBlock, 0, s>>>(e->d_item_covered, n_items, item_nnz, e->nnz, e->d_item_ids,
                                                                          e->d_pc);
    CU_TRY(e, cudaGetLastError());
    if (int rc = read_counters(e, &pc)) return rc;
    e->dense_own = offsets_used;   // tiles off the grid may overlap
    sddmm_b200_plan_info &p = e->plan;
    p.dense_tiles = n_dense;
    p.dense_nnz = static_cast<int64_t>(pc.dense_nnz);
    p.dense_tile_rows = p.dense_tile_cols = kDenseTile;
    e->n_residual_items = pc.residual_items;
    e->dense_fma = fp32;   // (the tensor-core modes are faster on theirs at every K: 50 and 59 us against 73 at K = 32)
    if (e->dense_fma) {
        int occ = 0;
        CU_TRY(e, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, dense_fma_function(e->dense_own), kFmaThreads, 0));
        if (occ < 1) return fail(e, SDDMM_B200_ERR_CUDA, "dense-tile FMA kernel does not fit on an SM");
        e->n_dense = n_dense;
        p.dense_block = kFmaThreads;
        p.dense_grid = std::min(n_dense, e->sm_count * occ);
        return SDDMM_B200_OK;
    }
    const bool split = e->mode == SDDMM_B200_FP32_TC;
    const int64_t kx = split ? 3 * e->K : e->K;
    int st = make_operand_map(e, &e->map_a, split ? e->d_Ax : e->d_A32, e->M, kx);
    if (!st) st = make_operand_map(e, &e->map_b, split ? e->d_Bx : e->d_B32, e->N, kx);
    if (st) return st;
    // fp32-grade mode, K >= 64: the three-slot operand scheme (measured on the 64 x 64-block configuration, K = 64 / 128:
    // 74 / 114 us against 93 / 160 us with one A block + one B block; K = 32: 63-66 us either way, the shared-memory data
    // pipe that the epilogue and the operand reads share is the limit there).  Knob "dense_split3": 0 = never, 1 = always.
    e->dense_split3 = split && (e->knob_dense_split3 > 0 || (e->knob_dense_split3 < 0 && e->K >= 64));
    const void *dense_fn = dense_function(e->dense_own, e->dense_split3);
    const uint32_t dense_smem = e->dense_split3 ? DenseSmemT<true>::kDynamicBytes : DenseSmemT<false>::kDynamicBytes;
    if (ensure_dynamic_smem_limit(dense_fn, e->device, dense_smem))
        return fail(e, SDDMM_B200_ERR_CUDA, "dense-tile kernel: cannot raise the dynamic shared memory limit");
    CU_TRY(e, cudaFuncSetAttribute(dense_fn, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared));
    e->n_dense = n_dense;
    p.dense_block = kDenseThreads;
    p.dense_smem_bytes = static_cast<int32_t>(dense_smem);
    // Resident CTAs per SM, from the kernel's own resources (the runtime's occupancy query answers 1 for this kernel):
    // shared memory (+1 KB the driver reserves per CTA), registers (allocated per warp in units of 256), tensor memory columns.
    cudaFuncAttributes fa;
    CU_TRY(e, cudaFuncGetAttributes(&fa, dense_fn));
    int smem_per_sm = 0, regs_per_sm = 0;   // (single attributes: the full property query takes milliseconds)
    CU_TRY(e, cudaDeviceGetAttribute(&smem_per_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, e->device));
    CU_TRY(e, cudaDeviceGetAttribute(&regs_per_sm, cudaDevAttrMaxRegistersPerMultiprocessor, e->device));
    const int by_smem = static_cast<int>(static_cast<size_t>(smem_per_sm) / (dense_smem + fa.sharedSizeBytes + 1024));
    const int regs_per_warp = ((fa.numRegs * 32 + 255) / 256) * 256;
    const int by_regs = regs_per_sm / (regs_per_warp * (kDenseThreads / 32));
    const int by_tmem = 512 / static_cast<int>(e->dense_split3 ? DenseSmemT<true>::kTmemColumns : DenseSmemT<false>::kTmemColumns);
    int dense_ctas_per_sm = std::min(std::min(by_smem, by_regs), std::min(by_tmem, kDenseCtasPerSm));
    if (dense_ctas_per_sm < 1) return fail(e, SDDMM_B200_ERR_CUDA, "dense-tile kernel does not fit on an SM");
    if (const char *env = getenv("SDDMM_B200_DENSE_CTAS_PER_SM")) {   // tuning knob: fewer resident CTAs per SM
        const int v = atoi(env);
        if (v >= 1 && v < dense_ctas_per_sm) dense_ctas_per_sm = v;
    }
    p.dense_grid = std::min((n_dense + 1) / 2, e->sm_count * dense_ctas_per_sm);
    return SDDMM_B200_OK;
}

// Validation + histogram + plan, after the operands are in the arena.
using RowGroupFn = void (*)(const RowGroupArgs);
RowGroupFn pick_rowgroup(int rows, int cpl) {
    if (cpl == 1) return rows == 2 ? sddmm_rowgroup_kernel<2, 1> : rows == 3 ? sddmm_rowgroup_kernel<3, 1> : sddmm_rowgroup_kernel<4, 1>;
    return rows == 2 ? sddmm_rowgroup_kernel<2, 2> : rows == 3 ? sddmm_rowgroup_kernel<3, 2> : sddmm_rowgroup_kernel<4, 2>;
}

using RowSegGroupFn = void (*)(const RowSegGroupArgs);
template <int LPR, int RUN, bool WHOLE>
RowSegGroupFn pick_rowseg_group_rows(int rows) {
    return rows == 2 ? sddmm_rowseg_group_kernel<LPR, 2, RUN, WHOLE> : rows == 3 ? sddmm_rowseg_group_kernel<LPR, 3, RUN, WHOLE> : sddmm_rowseg_group_kernel<LPR, 4, RUN, WHOLE>;
}
// lanes per row
int group_lanes(const sddmm_b200_engine *e) { return e->Ks <= 32 ? 4 : e->Ks <= 64 ? 8 : e->Ks <= 128 ? 16 : 32; }
// units that one group of lanes takes one after the other, see the kernel: rows of 64 and 128 elements, where every warp of the chip has
// two steps or more all the same (70 000 nonzeros in 3 x 3 blocks, K = 64: 11.7 us with one, 12.5 with two)
int group_run(const sddmm_b200_engine *e) {
    const int64_t warps = 2 * kRowSegWarps * static_cast<int64_t>(e->sm_count);
    return (e->Ks == 64 || e->Ks == 128) && e->n_units > 2 * warps * (256 / e->Ks) ? 2 : 1;
}
// rows of up to 256 elements, bf16 rows of 32, 64, 128, 192 or 256 (nullptr: no instantiation)
RowSegGroupFn pick_rowseg_group(const sddmm_b200_engine *e, int rows) {
    if (e->mode == SDDMM_B200_BF16) {
        switch (e->Ks) {
            case 32: return sddmm_rowseg_group_bf16_kernel<1, 16, 4>;
            case 64: return sddmm_rowseg_group_bf16_kernel<1, 32, 2>;
            case 128: return sddmm_rowseg_group_bf16_kernel<2, 32, 1>;
            case 192: return sddmm_rowseg_group_bf16_kernel<3, 32, 1>;
            case 256: return sddmm_rowseg_group_bf16_kernel<4, 32, 1>;
            default: return nullptr;
        }
    }
    if (e->Ks > 256 || e->Ks % 8 != 0) return nullptr;
    const bool whole = e->Ks == 8 * group_lanes(e);
    switch (group_lanes(e)) {
        case 4: return whole ? pick_rowseg_group_rows<4, 1, true>(rows) : pick_rowseg_group_rows<4, 1, false>(rows);
        case 8: return !whole ? pick_rowseg_group_rows<8, 1, false>(rows) : group_run(e) == 2 ? pick_rowseg_group_rows<8, 2, true>(rows) : pick_rowseg_group_rows<8, 1, true>(rows);
        case 16: return !whole ? pick_rowseg_group_rows<16, 1, false>(rows) : group_run(e) == 2 ? pick_rowseg_group_rows<16, 2, true>(rows) : pick_rowseg_group_rows<16, 1, true>(rows);
        default: return whole ? pick_rowseg_group_rows<32, 1, true>(rows) : pick_rowseg_group_rows<32, 1, false>(rows);
    }
}

using RowSegFn = void (*)(const RowSegArgs);

template <int TAIL, bool COPIES>   // (ragged rows of one piece always leave the product out)
RowSegFn pick_rowseg(int pieces) {
    switch (pieces) {
        case 1: return sddmm_rowseg_kernel<1, TAIL == kTail ? kTailSpecials : TAIL, COPIES, kWholeRows>;
        case 2: return sddmm_rowseg_kernel<2, TAIL, COPIES, kWholeRows>;
        case 3: return sddmm_rowseg_kernel<3, TAIL == kNoTail ? kTail : TAIL, COPIES, kWholeRows>;   // (see RowTail)
        case 4: return sddmm_rowseg_kernel<4, TAIL, COPIES, kWholeRows>;
        case 5: return sddmm_rowseg_kernel<5, TAIL, COPIES, kWholeRows>;
        case 6: return sddmm_rowseg_kernel<6, TAIL, COPIES, kWholeRows>;
        case 7: return sddmm_rowseg_kernel<7, TAIL, COPIES, kWholeRows>;
        default: return sddmm_rowseg_kernel<8, TAIL, COPIES, kWholeRows>;
    }
}
template <bool SPECIALS>
RowSegFn pick_rowseg_wide(int pieces) {   // (nullptr: an odd number of pieces)
    switch (pieces) {
        case 2: return sddmm_rowseg_wide_kernel<2, SPECIALS, kWholeRows>;
        case 4: return sddmm_rowseg_wide_kernel<4, SPECIALS, kWholeRows>;
        case 6: return sddmm_rowseg_wide_kernel<6, SPECIALS, kWholeRows>;
        case 8: return sddmm_rowseg_wide_kernel<8, SPECIALS, kWholeRows>;
        default: return nullptr;
    }
}
template <int TAIL, bool COPIES>
RowSegFn pick_rowseg_bf16(int64_t Ks) {
    if (Ks <= 32) return sddmm_rowseg_bf16_kernel<1, 16, 8, 3, COPIES && TAIL == kNoTail ? kTail : TAIL, COPIES>;   // (see RowTail)
    if (Ks <= 64) return sddmm_rowseg_bf16_kernel<1, 32, 8, 2, TAIL == kNoTail ? kTail : TAIL, COPIES>;   // (see RowTail)
    if (Ks <= 128) return sddmm_rowseg_bf16_kernel<2, 32, 4, 2, TAIL, COPIES>;
    if (Ks <= 192) return sddmm_rowseg_bf16_kernel<3, 32, 4, 1, TAIL, COPIES>;
    return sddmm_rowseg_bf16_kernel<4, 32, 2, 1, TAIL, COPIES>;
}
// a slice of K: without panels of a B that does not fit L2, the order that DRAM likes
template <int PIECES, int STEP>
RowSegFn pick_rowseg_slice(const sddmm_b200_engine *e, bool copies) {
    if (copies) return sddmm_rowseg_kernel<PIECES, kNoTail, true, STEP>;
    if (static_cast<double>(e->N) * (128.0 * PIECES) > e->l2_bytes) return sddmm_rowseg_wide_kernel<PIECES, false, STEP>;
    return sddmm_rowseg_kernel<PIECES, kNoTail, false, STEP>;
}
template <int PIECES>
RowSegFn pick_rowseg_slice(const sddmm_b200_engine *e, bool copies, SliceStep step) {
    return step == kFirstSlice ? pick_rowseg_slice<PIECES, kFirstSlice>(e, copies) : step == kNextSlice ? pick_rowseg_slice<PIECES, kNextSlice>(e, copies)
                                                                                                        : pick_rowseg_slice<PIECES, kLastSlice>(e, copies);
}
RowSegFn pick_rowseg_slice(const sddmm_b200_engine *e, bool copies, SliceStep step) {
    return e->slice_cols == 128 ? pick_rowseg_slice<4>(e, copies, step) : pick_rowseg_slice<2>(e, copies, step);
}
// The row-segment kernel instantiation for this engine's storage and K (`copies`: S values from the per-unit copies).
template <int TAIL>
RowSegFn seg_function_tail(const sddmm_b200_engine *e, bool copies) {
    if (e->mode == SDDMM_B200_BF16) return copies ? pick_rowseg_bf16<TAIL, true>(e->Ks) : pick_rowseg_bf16<TAIL, false>(e->Ks);
    const int pieces = static_cast<int>((e->Ks + 31) / 32);
    // whole rows of a B that does not fit L2, without panels (rows too short for them): the order that DRAM likes
    if (!copies && static_cast<double>(e->N) * e->Ks * 4.0 > e->l2_bytes)
        if (RowSegFn fn = pick_rowseg_wide<TAIL == kTailSpecials>(pieces)) return fn;
    return copies ? pick_rowseg<TAIL, true>(pieces) : pick_rowseg<TAIL, false>(pieces);
}
RowSegFn seg_function(const sddmm_b200_engine *e, bool copies) {
    if (e->mode != SDDMM_B200_BF16 && e->seg_slices > 1) return pick_rowseg_slice(e, copies, kLastSlice);
    if (leave_out_past_end(e)) return seg_function_tail<kTailSpecials>(e, copies);
    return ragged_rows(e) ? seg_function_tail<kTail>(e, copies) : seg_function_tail<kNoTail>(e, copies);
}
// persistent grid of a streaming kernel over `n_units` units, `per_step` of them per warp step
int seg_grid(sddmm_b200_engine *e, const void *fn, int warps, int per_step, int64_t n_units, int32_t *grid) {
    int occ = 0;
    CU_TRY(e, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, warps * 32, 0));
    if (occ < 1) return fail(e, SDDMM_B200_ERR_CUDA, "row-segment kernel does not fit on an SM");
    const int64_t steps = (n_units + per_step - 1) / per_step;
    *grid = static_cast<int32_t>(std::min<int64_t>((steps + warps - 1) / warps, static_cast<int64_t>(e->sm_count) * occ));
    return SDDMM_B200_OK;
}

// whether the list is ordered by size (plan_sizes.cuh), for the rows that one launch takes
bool list_by_size(const sddmm_b200_engine *e, int32_t long_rows) {
    const int64_t row = e->seg_slices > 1 ? e->slice_cols : e->Ks;
    return by_size(e->mode == SDDMM_B200_BF16, row, long_rows > 0, gathered_bytes(e, row), e->l2_bytes);
}

// Enqueue the kernel that writes the list, from tile sums that are there (scanned: as the units before each tile).
template <typename Runs, typename HDR>
int enqueue_build(sddmm_b200_engine *e, cudaStream_t s, const Runs &runs, int64_t n, bool scanned, int64_t cap, HDR *units, int32_t *unit_cols,
                  const ListGate &gate, bool by_size, const UnitValues &values) {
    const int tiles = static_cast<int>(unit_tiles(n));
    if constexpr (sizeof(HDR) == sizeof(int2)) {
        if (by_size) k_unit_build<Runs, HDR, true><<<tiles, kUnitBlock, 0, s>>>(runs, n, e->d_scan_tiles, cap, e->d_pc, units, unit_cols, scanned, gate, values);
        else k_unit_build<Runs, HDR, false><<<tiles, kUnitBlock, 0, s>>>(runs, n, e->d_scan_tiles, cap, e->d_pc, units, unit_cols, scanned, gate, values);
    } else {
        k_unit_build<Runs, HDR, false><<<tiles, kUnitBlock, 0, s>>>(runs, n, e->d_scan_tiles, cap, e->d_pc, units, unit_cols, scanned, gate, values);
    }
    CU_TRY(e, cudaGetLastError());
    return SDDMM_B200_OK;
}

// Enqueue the list over n entries; *units = how many there are goes to the plan counters.  have_sums: k_row_stats has left the tile
// sums and the total.
template <typename Runs, typename HDR>
int enqueue_units(sddmm_b200_engine *e, cudaStream_t s, const Runs &runs, int64_t n, bool have_sums, int64_t cap, HDR *units, int32_t *unit_cols,
                  const ListGate &gate = ListGate{}, bool by_size = false, const UnitValues &values = UnitValues{}) {
    const int tiles = static_cast<int>(unit_tiles(n));
    if (int rc = check_tile_sums(e, tiles)) return rc;
    if (!have_sums) {
        if constexpr (!Runs::kChosen) CU_TRY(e, cudaMemsetAsync(&e->d_pc->units, 0, sizeof(unsigned long long), s));
        else k_panel_cuts<<<grid_for(e->M, kUnitBlock, e->sm_count * 8), kUnitBlock, 0, s>>>(runs, e->d_pc, gate);
        k_unit_sums<<<tiles, kUnitBlock, 0, s>>>(runs, n, e->d_scan_tiles, e->d_pc, gate);
    }
    const bool scanned = tiles > kDirectTiles;
    if (scanned) k_scan_sums<<<1, kScanBlock, 0, s>>>(e->d_scan_tiles, tiles, &e->d_pc->units);
    return enqueue_build(e, s, runs, n, scanned, cap, units, unit_cols, gate, by_size, values);
}

// Gathers of B that have to disappear before row groups are taken: 30 % of all, and as many as are worth the planning.  What they save
// of a run is estimated at the rate of the L2 -> SM fabric (rows of less than a line at a line's; rows that leave lanes idle save
// less, K = 96, 3.7 M nonzeros: 34 us of 51).  What groups cost is a second look at the counters, the match and a list that cannot be
// built beside the column scan.
//   fp32: 30 to 50 us, so that a single run pays from about 45 us on.  Upload and run, without / with groups: K = 128, 1 / 2 / 3.7 M
//     nonzeros (18 / 37 / 67 us) 134 / 167, 178 / 181, 235 / 223 us; K = 256, 1 / 2 M (37 / 73) 167 / 170, 246 / 218; K = 96, 3.7 M (38) 205 / 230.
//   fp32 rows of 32 and 64: taken whatever they save.  These are what plans that are held and run again have counted on (without /
//     with, 1 M: K = 32 19.4 / 13.6 us a run, K = 64 25.7 / 16.4), and a single run, 122 / 160 and 124 / 160 us, is not slower than it was.
//   bf16: 5 to 15 us (no list is built early there, tiles are looked for first), back by the fourth run from 4 us on: K = 64, 1 / 2 /
//     3.7 M (4.6 / 9.2 / 17 us) 169 / 179, 193 / 202, 225 / 222 us, a held run 18 / 14, 28 / 19, 43 / 29.
// Knob "group_units" = 1: whatever they are worth.
double groups_from(const sddmm_b200_engine *e) {
    const bool bf = e->mode == SDDMM_B200_BF16;
    const double share = 0.3 * static_cast<double>(e->nnz);
    if (!e->use_seg || e->knob_group_units >= 0 || (!bf && (e->Ks == 32 || e->Ks == 64))) return share;
    const double bytes = std::max(128.0, static_cast<double>(e->Ks) * static_cast<double>(elem_bytes(e)));
    const double used = bf || e->Ks <= 32 ? 1.0 : static_cast<double>(e->Ks) / (8.0 * group_lanes(e));   // of a row's lanes
    return std::max(share, (bf ? 4.0 : 45.0) * 18.6e6 / (bytes * used));
}

bool group_possible(const sddmm_b200_engine *e) {
    if (0.75 * static_cast<double>(e->nnz) < groups_from(e)) return false;   // (groups of four rows throughout)
    if ((e->flags & SDDMM_B200_FLAG_NO_ROW_GROUPS) || e->M < 4) return false;
    if (e->knob_group_units != 0 && e->use_seg) return pick_rowseg_group(e, 2) != nullptr;
    return e->mode != SDDMM_B200_BF16 && (e->K == 32 || e->K == 64);
}
// candidates: G = 2, 3, 4 rows per group, first full group starting at row 0 .. G-1 (counters slot = G(G-1)/2 - 1 + first)
int group_slot(int G, int first) { return G * (G - 1) / 2 - 1 + first; }
// G and `first` are chosen on a sample of the groups (about 8 000 rows' worth, at most 1 in 64 of them); the chosen grouping is then matched exactly.
// (At most 1 in 16, every upload of a large matrix pays: 2.6 M rows 51 us, 1 in 64 19.)
int group_sample(const sddmm_b200_engine *e) { return static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(64, e->M / 8192))); }
int enqueue_group_sample(sddmm_b200_engine *e) {
    const int every = group_sample(e);
    const dim3 grid(grid_for((e->M / 2 / every + 2) * 32, kBlock, e->sm_count * 2), 9);
    k_group_match<<<grid, kBlock, 0, e->stream>>>(e->d_rp, e->d_col, static_cast<int32_t>(e->M), static_cast<int32_t>(e->nnz), 0, 0, every, nullptr,
                                                  e->d_pc->group_cover, e->d_pc->group_count);
    CU_TRY(e, cudaGetLastError());
    return SDDMM_B200_OK;
}

// Row groups: groups of 2, 3 or 4 consecutive rows with one column list (first full group at row 0 .. G-1) share each gather of B.
// The path is taken (for the whole matrix) when it removes at least 30 % of the gathers; K <= 256.
// base_pc: counters that include enqueue_group_sample's.
int build_rowgroup_plan(sddmm_b200_engine *e, const PlanCounters &base_pc) {
    if (!group_possible(e) || base_pc.max_row_nnz > kGroupRowMax) return SDDMM_B200_OK;
    cudaStream_t s = e->stream;
    const int every = group_sample(e);
    const int32_t M = static_cast<int32_t>(e->M), nnz = static_cast<int32_t>(e->nnz);
    int bs = 0;
    if (group_saving(base_pc.group_cover, every, &bs) < groups_from(e)) return SDDMM_B200_OK;
    const int best = bs < 2 ? 2 : bs < 5 ? 3 : 4, best_first = bs - group_slot(best, 0);
    const int32_t n_groups = group_count(M, best, best_first);
    const bool units = e->knob_group_units != 0 && e->use_seg;
    e->group_tried = true;
    // exact match of the chosen grouping, and -- speculating that the sample was right -- the unit list over it
    CU_TRY(e, cudaMemsetAsync(&e->d_pc->group_cover[bs], 0, sizeof(unsigned long long), s));
    CU_TRY(e, cudaMemsetAsync(&e->d_pc->group_count[bs], 0, sizeof(int), s));
    k_group_match<<<grid_for(static_cast<int64_t>(n_groups) * 32, kBlock, e->sm_count * 8), kBlock, 0, s>>>(
        e->d_rp, e->d_col, M, nnz, best, best_first, 1, e->d_group_ok, &e->d_pc->group_cover[bs], &e->d_pc->group_count[bs]);
    if (units) {
        const RunsOfGroups runs{e->d_rp, e->d_col, M, nnz, best, best_first, e->d_group_ok};
        if (int rc = enqueue_units(e, s, runs, e->M, false, e->unit_cap, reinterpret_cast<int4 *>(e->d_units), e->d_unit_cols)) return rc;
    }
    CU_TRY(e, cudaGetLastError());
    PlanCounters pc;
    if (int rc = read_counters(e, &pc)) return rc;
    if (static_cast<double>(pc.group_cover[bs]) * (1.0 - 1.0 / best) < 0.3 * static_cast<double>(e->nnz)) return SDDMM_B200_OK;   // the sample overestimated
    sddmm_b200_plan_info &p = e->plan;
    if (units) {
        if (pc.units == 0 || pc.units > static_cast<unsigned long long>(std::min<int64_t>(e->unit_cap, kUnitLimit)))
            return fail(e, SDDMM_B200_ERR_CUDA, "row-group plan: %llu units for a list of %lld", pc.units, (long long)e->unit_cap);
        e->n_units = static_cast<int32_t>(pc.units);
        const int per_step = e->mode == SDDMM_B200_BF16 ? 8 : 32 / group_lanes(e) * group_run(e);
        if (int rc = seg_grid(e, reinterpret_cast<const void *>(pick_rowseg_group(e, best)), kRowSegWarps, per_step, e->n_units, &p.rowgroup_grid)) return rc;
        p.rowseg_units = e->n_units;
        p.rowseg_panels = 1;
    } else {
        RowGroupFn fn = pick_rowgroup(best, static_cast<int>(e->K / 32));
        int occ = 0;
        CU_TRY(e, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, kRowGroupWarps * 32, 0));
        if (occ < 1) return fail(e, SDDMM_B200_ERR_CUDA, "row-group kernel does not fit on an SM");
        p.rowgroup_grid = std::min((n_groups + kRowGroupWarps - 1) / kRowGroupWarps, e->sm_count * occ);
    }
    if (units && e->slice_major) {   // (whole rows here)
        e->slice_major = false;
        if (e->Ks == e->K) e->d_Ap = e->d_Bp = nullptr;
    }
    e->rg_rows = best;
    e->rg_first = best_first;
    e->rg_groups = n_groups;
    e->rg_units = units;
    p.rowgroup_nnz = static_cast<int64_t>(pc.group_cover[bs]);
    p.rowgroup_groups = pc.group_count[bs];
    p.rowgroup_rows = best;
    p.rowtile_nnz = 0;
    p.rowtile_items = 0;
    p.n_kernels = 1;
    return SDDMM_B200_OK;
}

// What the dense tiles left, as row segments: the uncovered runs of every row cut into units, so that the residual
// kernel touches only those nonzeros (a kernel that walks all work items and skips the covered nonzeros costs as much as
// the whole matrix when the tiles leave a little in every item).
int build_residual_units(sddmm_b200_engine *e) {
    if (!e->use_seg) return SDDMM_B200_OK;
    const int32_t M = static_cast<int32_t>(e->M);
    const int n_tiles = static_cast<int>(scan_tiles(e->M));
    if (int rc = check_tile_sums(e, n_tiles)) return rc;
    const int cap = e->sm_count * 32;
    cudaStream_t s = e->stream;
    k_residual_unit_count<<<grid_for(e->M * 32, kBlock, cap), kBlock, 0, s>>>(e->d_rp, M, e->d_covered, e->d_unit_off);
    k_scan_tile_sums<<<n_tiles, kScanBlock, 0, s>>>(e->d_unit_off, e->M, e->d_scan_tiles);
    k_scan_sums<<<1, kScanBlock, 0, s>>>(e->d_scan_tiles, n_tiles, &e->d_pc->units);
    k_scan_apply<<<n_tiles, kScanBlock, 0, s>>>(e->d_unit_off, e->M, e->d_scan_tiles);
    CU_TRY(e, cudaGetLastError());
    PlanCounters pc;
    if (int rc = read_counters(e, &pc)) return rc;
    if (pc.units == 0 || pc.units > static_cast<unsigned long long>(e->unit_cap))   // (more is not possible: unit_capacity)
        return fail(e, SDDMM_B200_ERR_CUDA, "residual plan: %llu units for a list of %lld", pc.units, (long long)e->unit_cap);
    k_residual_unit_fill<<<grid_for(e->M * 32, kBlock, cap), kBlock, 0, s>>>(e->d_rp, M, e->d_covered, e->d_unit_off, e->d_col, e->d_units, e->d_unit_cols);
    k_unit_pad<<<1, 64, 0, s>>>(e->d_units, e->d_unit_cols, e->d_pc, e->unit_cap);
    CU_TRY(e, cudaGetLastError());
    e->n_units = static_cast<int32_t>(pc.units);
    e->seg_residual = true;
    e->plan.rowseg_units = e->n_units;
    e->plan.rowseg_panels = 1;
    e->plan.rowseg_passes = e->seg_slices;
    return seg_grid(e, reinterpret_cast<const void *>(seg_function(e, false)), kRowSegWarps, 8, e->n_units, &e->plan.rowseg_grid);
}

// The forms of the list over the whole matrix
ListForms list_forms(const sddmm_b200_engine *e) {
    ListForms f;
    f.plain = e->panels_plain;
    f.plain_cols = static_cast<int32_t>((e->N + f.plain - 1) / f.plain);
    f.plain_for_8 = e->nnz < 16 * e->M && e->knob_panels < 1;
    f.plain_by_size = list_by_size(e, 0);
    if (e->long_threshold > 0) {
        f.longs = e->panels_long;
        f.long_cols = static_cast<int32_t>((e->N + f.longs - 1) / f.longs);
        f.long_rows = e->long_threshold;
        f.long_always = e->knob_long_rows >= 0;
        f.long_by_size = list_by_size(e, f.long_rows);
    }
    return f;
}

// Enqueue the list over the whole matrix.  have_sums: k_row_stats has left the tile sums of whole rows.
int enqueue_unit_list(sddmm_b200_engine *e, cudaStream_t s, const ListForms &forms, bool have_sums, const ListGate &gate = ListGate{},
                      const UnitValues &values = UnitValues{}) {
    const int32_t M = static_cast<int32_t>(e->M), nnz = static_cast<int32_t>(e->nnz);
    int st;
    if (forms.plain > 1 || forms.long_rows > 0) {
        // (the starts of the panels: in the half of the headers' memory that plain units leave)
        const RunsOfForms runs{e->d_rp, e->d_col, M, nnz, forms, reinterpret_cast<int32_t *>(e->d_units + e->unit_cap + 8), 2 * (e->unit_cap + 8),
                               have_sums, have_sums};
        int64_t most = e->M;   // entries of the form with the most tiles: the grid is made for that one
        for (const int64_t n : {e->M * forms.plain, forms.long_rows > 0 ? e->M * (forms.longs + 1) : 0})
            if (unit_tiles(n) > unit_tiles(most)) most = n;
        st = enqueue_units(e, s, runs, most, false, e->unit_cap, e->d_units, e->d_unit_cols, gate,
                           (!have_sums && forms.plain_by_size) || forms.long_by_size, values);
        if (!st && have_sums) {
            const WholeRowsOfForms whole{RunsOfRows{e->d_rp, e->d_col, M, nnz}, forms};
            st = enqueue_build(e, s, whole, e->M, unit_tiles(most) > kDirectTiles, e->unit_cap, e->d_units, e->d_unit_cols, gate, forms.plain_by_size, UnitValues{});
        }
    } else {
        const RunsOfRows runs{e->d_rp, e->d_col, M, nnz};
        st = enqueue_units(e, s, runs, e->M, have_sums, e->unit_cap, e->d_units, e->d_unit_cols, gate, forms.plain_by_size);
    }
    if (st) return st;
    if (e->mode == SDDMM_B200_BF16) k_unit_pad<<<1, 64, 0, s>>>(e->d_units, e->d_unit_cols, e->d_pc, e->unit_cap);
    CU_TRY(e, cudaGetLastError());
    return SDDMM_B200_OK;
}

// Row segments over the whole matrix.  early: the forms of the list that is already there, counted in pc (null: none); early_values:
// with the copies of the S values.
int build_rowseg_plan(sddmm_b200_engine *e, PlanCounters pc, const ListForms *early, bool early_values) {
    e->seg_copies = false;
    e->n_units = 0;
    if (!e->use_seg) return SDDMM_B200_OK;
    auto choose = [&]() -> ListForms::Choice {
        ListForms f = list_forms(e);
        if (pc.unsorted_cols) {   // (a panel run is a contiguous piece of a row only when its columns are sorted)
            f.plain = 1;
            f.long_rows = 0;
        }
        return f.choose(&pc, e->nnz);
    };
    ListForms::Choice c = choose();
    if (e->slice_major && e->knob_k_slices < 0 && (c.long_rows > 0 || pc.unsorted_cols || e->panels_plain == 1)) {
        e->slice_major = false;   // (slices_apart: the copies pay with plain panels only)
        if (e->Ks == e->K) e->d_Ap = e->d_Bp = nullptr;
        choose_list_forms(e);
        c = choose();
    }
    if (e->knob_k_slices < 0 && e->K <= 256) {
        if (c.long_rows > 0 && long_rows_whole(e)) e->seg_slices = 1;
        // slices of 64 that do not fit L2 and get no panels either: whole rows
        if (c.panels == 1 && e->slice_cols == 64 && e->nnz < 16 * e->M && gathered_bytes(e, 64) > e->l2_bytes) e->seg_slices = 1;
    }
    bool built = false;
    e->values_built = false;
    if (early) {
        const ListForms::Choice was = early->choose(&pc, e->nnz);
        built = was.panels == c.panels && was.long_rows == c.long_rows && (c.panels == 1 || was.panel_cols == c.panel_cols);
        e->values_built = built && early_values;
    }
    if (!built) {
        ListForms f;   // the one form
        f.plain = c.long_rows > 0 ? 1 : c.panels;
        f.plain_cols = f.long_cols = c.panel_cols;
        f.longs = c.panels - 1;
        f.long_rows = c.long_rows;
        f.long_always = true;
        f.plain_by_size = f.long_by_size = list_by_size(e, c.long_rows);
        if (int rc = enqueue_unit_list(e, e->stream, f, false)) return rc;
        if (int rc = read_counters(e, &pc)) return rc;
    }
    e->seg_copies = c.panels > 1;
    if (pc.units == 0 || pc.units > static_cast<unsigned long long>(std::min<int64_t>(e->unit_cap, kUnitLimit)))
        return fail(e, SDDMM_B200_ERR_CUDA, "row-segment plan: %llu units for a list of %lld", pc.units, (long long)e->unit_cap);
    e->n_units = static_cast<int32_t>(pc.units);
    sddmm_b200_plan_info &p = e->plan;
    p.rowseg_nnz = e->nnz;
    p.rowseg_units = e->n_units;
    p.rowseg_panels = c.panels;
    p.rowseg_passes = e->seg_slices;
    p.rowtile_nnz = 0;
    p.rowtile_items = 0;
    p.n_kernels = 1;
    return seg_grid(e, reinterpret_cast<const void *>(seg_function(e, e->seg_copies)), kRowSegWarps, 8, e->n_units, &p.rowseg_grid);
}

// Validation + statistics + plan.  join_copies: order the rest of the upload (copies on the side stream, conversions) before
// the first read-back, so that one wait of the host covers both.
int build_plan(sddmm_b200_engine *e, int item_nnz, int n_items, bool join_copies) {
    const int cap = e->sm_count * 8;
    cudaStream_t s = e->stream;
    CU_TRY(e, cudaMemsetAsync(e->d_pc, 0, e->plan_clear_bytes, s));   // counters, distinct columns, row-start bits
    e->n_dense = 0;
    e->n_units = 0;
    e->rg_rows = 0;
    e->seg_copies = false;
    e->group_tried = false;
    e->copies_joined = false;
    if (e->d_coo_rows)   // (rows out of order or out of range are counted, and every later kernel checks the bounds it gets from row_ptr)
        k_coo_to_row_ptr<<<grid_for(e->nnz + 1, kBlock, cap), kBlock, 0, s>>>(e->d_coo_rows, e->nnz, static_cast<int32_t>(e->M),
                                                                              e->coo_row_base, e->d_rp, e->d_pc);
    // What will most likely run is enqueued before anything is read back: the unit list, in the form that the row statistics choose on
    // the device (not where tiles decide first, or whether the copies of B are made slice by slice), and the sample that looks for row groups.
    const bool tiles_first = e->dense_possible && e->mode != SDDMM_B200_FP32;   // (fp32 mode: tiles are the exception)
    const ListForms forms = list_forms(e);
    const bool whole_rows = forms.plain == 1 && forms.long_rows == 0;
    const bool early_list = e->use_seg && !tiles_first && (whole_rows || !e->slice_major) && e->nnz > 0;
    const bool sums_beside = early_list && forms.plain == 1;
    k_row_stats<<<static_cast<int>(unit_tiles(e->M)), kUnitBlock, 0, s>>>(e->d_rp, static_cast<int32_t>(e->M), e->nnz, e->d_rowstart,
                                                                                            sums_beside ? e->d_scan_tiles : nullptr, e->d_pc);
    // The list needs the row statistics only: where the operands come from this GPU's memory it is built on the side
    // stream, behind their copies, while the columns are looked at here (each of the three kernels leaves much of the chip idle: 5.2 M
    // nonzeros, K = 64, upload and run 272 -> 256 us; 4 M, power law, 266 -> 249).  Not for rows long enough to lie in 64-wide tiles,
    // where the count of the column scan may make the list unnecessary (18 M in 64 x 64 blocks, upload 489 us, 572 with the list aside).
    // (Panels of columns that turn out not to be sorted may be runs that overlap, at most the whole row in each: their sums fit 32 bits.)
    const int64_t most_units = std::max<int64_t>(forms.plain, forms.longs + 1) * (e->nnz / 8 + e->M);
    const bool list_aside = early_list && join_copies && e->nnz < 64 * e->M && most_units < (int64_t(1) << 31);
    // The sample of the row groups comes behind the column scan: between it and the row statistics the sample waits for the copies'
    // kernels to end, and the scan with it (37 M nonzeros, bf16: 90 us), and before the list aside it delays that one (5.2 M, K = 64,
    // upload and run 244 -> 251).  A list behind it leaves its place to the groups' where the sample has found them.
    const bool groups = e->nnz > 0 && group_possible(e);
    ListGate gate;
    if (list_aside) {
        CU_TRY(e, cudaEventRecord(e->ev_fork, s));
        CU_TRY(e, cudaStreamWaitEvent(e->side_stream, e->ev_fork, 0));
        gate.columns_scanned = false;
        if (int rc = enqueue_unit_list(e, e->side_stream, forms, sums_beside, gate, UnitValues{e->d_sval, e->d_unit_sval})) return rc;
        CU_TRY(e, cudaEventRecord(e->ev_join, e->side_stream));
    }
    if (e->nnz > 0) {
        const size_t bitmap = (static_cast<size_t>(e->N) + 31) / 32 * 4;
        const int scan_blocks = grid_for(e->nnz, 4 * kColScanThreads, e->sm_count * 2);
        if (bitmap <= kColScanLocalBytes) {
            if (ensure_dynamic_smem_limit(reinterpret_cast<const void *>(k_col_scan<true>), e->device, kColScanLocalBytes))
                return fail(e, SDDMM_B200_ERR_CUDA, "column scan: cannot raise the dynamic shared memory limit");
            k_col_scan<true><<<std::min(scan_blocks, e->sm_count), kColScanThreads, bitmap, s>>>(e->d_col, e->nnz, static_cast<int32_t>(e->N), e->d_rowstart, e->d_touched, e->d_pc);
        } else {
            k_col_scan<false><<<scan_blocks, kColScanThreads, 0, s>>>(e->d_col, e->nnz, static_cast<int32_t>(e->N), e->d_rowstart, e->d_touched, e->d_pc);
        }
        CU_TRY(e, cudaGetLastError());
        if (groups)
            if (int rc = enqueue_group_sample(e)) return rc;
        if (early_list && !list_aside) {
            if (groups) {
                gate.groups_from = groups_from(e);
                gate.every = group_sample(e);
            }
            // (fp32 mode: tiles will most likely be looked for, and found, when the column scan's count is high enough)
            if (e->dense_possible && e->knob_offset_tiles <= 0) gate.tile_hint = (static_cast<unsigned long long>(e->nnz) + kTileHintShare - 1) / kTileHintShare;
            if (int rc = enqueue_unit_list(e, s, forms, sums_beside, gate)) return rc;
        }
    }
    if (list_aside) CU_TRY(e, cudaStreamWaitEvent(s, e->ev_join, 0));
    CU_TRY(e, cudaGetLastError());
    if (join_copies && !tiles_first && !e->slice_major) {
        CU_TRY(e, cudaStreamWaitEvent(s, e->ev_h2d, 0));
        if (int rc = convert_storage(e)) return rc;
        e->copies_joined = true;
    }
    PlanCounters pc;
    if (int rc = read_counters(e, &pc)) return rc;
    if (pc.bad_coo) return fail(e, SDDMM_B200_ERR_INDEX, "COO row indices must be sorted and inside [0, M)");
    if (pc.bad_row_ptr) return fail(e, SDDMM_B200_ERR_INDEX, "row_ptr must start at 0, end at nnz and be non-decreasing");
    const bool list_built = early_list && pc.list_built != 0;
    if (pc.bad_col) return fail(e, SDDMM_B200_ERR_INDEX, "column index outside [0, N)");

    sddmm_b200_plan_info &p = e->plan;
    std::memset(&p, 0, sizeof(p));
    p.rows = e->M; p.cols = e->N; p.k = e->K; p.nnz = e->nnz;
    p.rows_nonempty = static_cast<int64_t>(pc.rows_nonempty);
    p.cols_touched = static_cast<int64_t>(pc.cols_touched);
    p.max_row_nnz = pc.max_row_nnz;
    for (int b = 0; b < SDDMM_B200_HIST_BINS; ++b) p.row_len_hist[b] = static_cast<int64_t>(pc.hist[b]);
    p.cols_sorted = pc.unsorted_cols ? 0 : 1;
    p.mode = e->mode;
    p.n_devices = 1;

    // ---- row-tile kernel launch shape -----------------------------------------
    const size_t eb = elem_bytes(e);
    e->cpl = round_up_cpl(e->K);
    e->use_scalar = (e->K % 4 != 0) || e->cpl == 0 || static_cast<size_t>(e->K) * eb > kMaxStageBytes;
    p.rowtile_item_nnz = item_nnz;
    p.rowtile_block = kBlock;
    e->n_dense = 0;
    e->n_residual_items = n_items;
    if (e->nnz == 0) {
        p.n_kernels = 0;
        return SDDMM_B200_OK;
    }
    e->seg_residual = false;
    if (e->dense_possible) {
        int st = build_dense_plan(e, pc, item_nnz, n_items);
        if (st) return st;
        if (e->n_dense > 0 && e->n_residual_items > 0) {
            st = build_residual_units(e);
            if (st) return st;
        }
    }
    if (e->n_dense == 0) {
        int st = build_rowgroup_plan(e, pc);
        if (st) return st;
        if (e->rg_rows) return SDDMM_B200_OK;
        // (a grouping that was tried and dropped has used the list's memory)
        st = build_rowseg_plan(e, pc, list_built && !e->group_tried ? &forms : nullptr, list_aside);
        if (st) return st;
        if (e->use_seg) return SDDMM_B200_OK;
    }
    p.rowtile_nnz = e->nnz - p.dense_nnz;
    p.rowtile_items = e->n_residual_items;
    const int dense_kernels = e->n_dense > 0 ? 1 : 0;
    if (e->n_residual_items == 0) {
        p.n_kernels = dense_kernels;
        return SDDMM_B200_OK;
    }
    if (e->seg_residual) {   // the row-segment kernel computes what the tiles left
        p.rowseg_nnz = p.rowtile_nnz;
        p.rowtile_nnz = 0;
        p.rowtile_items = 0;
        p.n_kernels = 1 + dense_kernels;
        return SDDMM_B200_OK;
    }
    if (!e->use_scalar)
        k_item_rows<<<grid_for(n_items, kBlock, 1 << 30), kBlock, 0, s>>>(e->d_rp, static_cast<int32_t>(e->M), e->nnz, item_nnz, n_items,
                                                                          e->d_item_rows);
    if (e->use_scalar) {
        p.rowtile_rows_per_stage = 0;
        p.rowtile_smem_bytes = 0;
        p.rowtile_grid = grid_for(e->nnz, kBlock, e->sm_count * 8);
        p.n_kernels = 1;
        return SDDMM_B200_OK;
    }
    const double mean_len = static_cast<double>(e->nnz) / static_cast<double>(std::max<int64_t>(1, p.rows_nonempty));
    int64_t R = static_cast<int64_t>(item_nnz / std::max(1.0, mean_len)) + 1;
    R = (R + 7) / 8 * 8;
    const int64_t r_max = std::max<int64_t>(1, static_cast<int64_t>(kMaxStageBytes / (static_cast<size_t>(e->K) * eb)));
    R = std::max<int64_t>(1, std::min<int64_t>(std::min<int64_t>(R, r_max), e->M));
    p.rowtile_rows_per_stage = static_cast<int32_t>(R);
    p.rowtile_smem_bytes = static_cast<int32_t>(rowtile_smem_bytes(static_cast<int>(R), static_cast<uint32_t>(e->K * eb)));

    const void *fn = (e->mode == SDDMM_B200_BF16) ? reinterpret_cast<const void *>(pick_rowtile<__nv_bfloat16>(e->cpl, e->K == 32 * e->cpl))
                                                  : reinterpret_cast<const void *>(pick_rowtile<float>(e->cpl, e->K == 32 * e->cpl));
    if (ensure_dynamic_smem_limit(fn, e->device, kRowTileMaxSmem)) return fail(e, SDDMM_B200_ERR_CUDA, "row-tile kernel: cannot raise the dynamic shared memory limit");
    int occ = 0;
    CU_TRY(e, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, kBlock, p.rowtile_smem_bytes));
    if (occ < 1) return fail(e, SDDMM_B200_ERR_CUDA, "row-tile kernel does not fit on an SM (smem %d B)", p.rowtile_smem_bytes);
    p.rowtile_grid = std::min(e->n_residual_items, e->sm_count * occ);
    p.n_kernels = 1 + dense_kernels;
    return SDDMM_B200_OK;
}

int check_dims(sddmm_b200_engine *e, int64_t M, int64_t N, int64_t K, int64_t nnz) {
    if (M < 1 || N < 1 || K < 1 || nnz < 0) return fail(e, SDDMM_B200_ERR_ARG, "need M, N, K >= 1 and nnz >= 0");
    if (M >= (int64_t(1) << 31) - 1 || N >= (int64_t(1) << 31) - 1 || nnz >= (int64_t(1) << 31) - 8192)
        return fail(e, SDDMM_B200_ERR_ARG, "int32 index range exceeded");
    return SDDMM_B200_OK;
}

int cuda_status(sddmm_b200_engine *e, cudaError_t err) {
    CU_TRY(e, err);
    return SDDMM_B200_OK;
}

// all copies of an upload: pattern on the main stream, then values and dense operands on the side stream; ev_h2d after the last
int enqueue_copies(sddmm_b200_engine *e, const int32_t *row_ptr, const int32_t *coo_rows, const int32_t *col_idx, const float *s_val,
                   const float *A, const float *B, cudaMemcpyKind kind) {
    cudaStream_t s = e->stream, s2 = e->side_stream;
    const int64_t M = e->M, N = e->N, K = e->K, nnz = e->nnz;
    // (host sources: pageable memory is staged through pinned buffers by a pool of host threads, see host_staging.cuh)
    auto copy_in = [&](void *dst, const void *src, size_t bytes, cudaStream_t st, HostStager &stg) -> cudaError_t {
        return kind == cudaMemcpyHostToDevice ? stg.upload(dst, src, bytes, st) : cudaMemcpyAsync(dst, src, bytes, kind, st);
    };
    if (row_ptr) CU_TRY(e, copy_in(e->d_rp, row_ptr, static_cast<size_t>(M + 1) * 4, s, e->stager));
    if (coo_rows && nnz) CU_TRY(e, copy_in(e->d_coo_rows, coo_rows, static_cast<size_t>(nnz) * 4, s, e->stager));
    if (nnz) CU_TRY(e, copy_in(e->d_col, col_idx, static_cast<size_t>(nnz) * 4, s, e->stager));
    CU_TRY(e, cudaEventRecord(e->ev_join, s));
    CU_TRY(e, cudaStreamWaitEvent(s2, e->ev_join, 0));   // keeps the link order: pattern first
    if (nnz) CU_TRY(e, copy_in(e->d_sval, s_val, static_cast<size_t>(nnz) * 4, s2, e->stager2));
    CU_TRY(e, copy_in(e->d_A32, A, static_cast<size_t>(M * K) * 4, s2, e->stager2));
    if (e->B_on_device) CU_TRY(e, cudaMemcpyAsync(e->d_B32, e->B_on_device, static_cast<size_t>(N * K) * 4, cudaMemcpyDeviceToDevice, s2));
    else CU_TRY(e, copy_in(e->d_B32, B, static_cast<size_t>(N * K) * 4, s2, e->stager2));
    CU_TRY(e, cudaEventRecord(e->ev_h2d, s2));
    if (e->on_copies_enqueued) e->on_copies_enqueued(e->on_copies_user);
    return SDDMM_B200_OK;
}

int upload_common(sddmm_b200_engine *e, int64_t M, int64_t N, int64_t K, int64_t nnz, const int32_t *row_ptr,
                  const int32_t *coo_rows, const int32_t *col_idx, const float *s_val, const float *A, const float *B,
                  cudaMemcpyKind kind) {
    e->uploaded = false;
    e->ran = false;
    e->spmm_units = 0;
    drop_graph(e);
    e->M = M; e->N = N; e->K = K; e->nnz = nnz;
    const int item_nnz = choose_item_nnz(e);
    const int n_items = static_cast<int>((nnz + item_nnz - 1) / item_nnz);
    if (e->mode == SDDMM_B200_BF16 && (K % 8 != 0 || K > 256))
        return fail(e, SDDMM_B200_ERR_UNSUPPORTED, "bf16 storage needs K %% 8 == 0 and K <= 256 (K = %lld)", (long long)K);
    int st = carve_arena(e, coo_rows != nullptr, n_items, kFull);
    if (st == SDDMM_B200_ERR_OOM && e->d_Ap_wanted) st = carve_arena(e, coo_rows != nullptr, n_items, kNoCopies);
    if (st == SDDMM_B200_ERR_OOM && e->use_seg) st = carve_arena(e, coo_rows != nullptr, n_items, kNoLists);
    if (st) return st;
    // The pattern goes first, on the main stream, and is planned there while S.val, A and B -- which the plan does not read -- still
    // cross the host link on the side stream.  (Copies from pageable memory are staged by the calling thread, which launches the plan
    // after them: there the plan is not hidden.)
    cudaStream_t s = e->stream, s2 = e->side_stream;
    if (e->h2d_after) CU_TRY(e, cudaStreamWaitEvent(s, e->h2d_after, 0));
    st = enqueue_copies(e, row_ptr, coo_rows, col_idx, s_val, A, B, kind);
    if (!st) st = build_plan(e, item_nnz, n_items, kind == cudaMemcpyDeviceToDevice);
    if (!st && !e->copies_joined) {
        st = cuda_status(e, cudaStreamWaitEvent(s, e->ev_h2d, 0));
        if (!st) st = convert_storage(e);
    } else if (!st && !e->values_built) {
        st = refresh_unit_values(e);   // (the list was not there yet)
    }
    if (!st) st = cuda_status(e, cudaStreamSynchronize(s));   // the caller's buffers are free again when this returns
    if (st) {   // nothing of a failed upload may still be reading the caller's buffers
        cudaStreamSynchronize(s2);
        cudaStreamSynchronize(s);
        if (e->B_on_device == e->b_stage) e->B_on_device = nullptr;
        return st;
    }
    if (e->B_on_device == e->b_stage) e->B_on_device = nullptr;
    settle_specials(e);
    e->uploaded = true;
    return SDDMM_B200_OK;
}

// Where the kernels of a run go: onto the engine's two streams, or, as nodes, into a graph.  (The graph is put together node by
// node and not by stream capture: while any stream of a device is being captured, another thread's cudaDeviceSynchronize fails, and
// ends the capture.)
struct RunTarget {
    sddmm_b200_engine *e;
    cudaGraph_t graph;                               // null: the streams
    cudaGraphNode_t last[2] = {nullptr, nullptr};    // of the main and the side stream's kernels
    template <typename T>
    struct Same { using type = T; };
    template <typename... P>
    cudaError_t launch(bool side, void (*fn)(P...), int grid, int block, size_t smem, typename Same<P>::type... args) {
        void *params[] = {&args...};
        if (!graph) return cudaLaunchKernel(reinterpret_cast<const void *>(fn), dim3(grid), dim3(block), params, smem, side ? e->side_stream : e->stream);
        cudaKernelNodeParams n = {};
        n.func = reinterpret_cast<void *>(fn);
        n.gridDim = dim3(grid);
        n.blockDim = dim3(block);
        n.sharedMemBytes = static_cast<unsigned>(smem);
        n.kernelParams = params;
        cudaGraphNode_t &before = last[side], node;
        const cudaError_t st = cudaGraphAddKernelNode(&node, graph, before ? &before : nullptr, before ? 1 : 0, &n);
        if (st == cudaSuccess) before = node;
        return st;
    }
};

// events right before / right after kernel number `kernels_launched`, on the stream it is launched on
int begin_kernel(sddmm_b200_engine *e, cudaStream_t st) {
    if (!e->kernel_timing) return SDDMM_B200_OK;   // a timing event between two launches costs microseconds: only on request
    CU_TRY(e, cudaEventRecord(e->ev_begin[e->kernels_launched], st));
    return SDDMM_B200_OK;
}
int mark_kernel(sddmm_b200_engine *e, const char *name, cudaStream_t st) {
    CU_TRY(e, cudaGetLastError());
    const int idx = e->kernels_launched;
    e->kernel_name[idx] = name;
    if (e->kernel_timing) CU_TRY(e, cudaEventRecord(e->ev_end[idx], st));
    e->kernels_launched = idx + 1;
    return SDDMM_B200_OK;
}

// the rows of A and B as the row-segment kernels read them
const void *seg_rows_a(const sddmm_b200_engine *e) { return e->mode == SDDMM_B200_BF16 ? static_cast<const void *>(e->d_A16) : e->d_Ap ? e->d_Ap : e->d_A32; }
const void *seg_rows_b(const sddmm_b200_engine *e) { return e->mode == SDDMM_B200_BF16 ? static_cast<const void *>(e->d_B16) : e->d_Bp ? e->d_Bp : e->d_B32; }

// the row-segment kernel over the engine's unit list (the whole matrix, or what the dense tiles left)
int launch_rowseg(sddmm_b200_engine *e, RunTarget &to, bool side, float *p_val) {
    cudaStream_t stream = side ? e->side_stream : e->stream;
    const sddmm_b200_plan_info &p = e->plan;
    RowSegArgs g;
    g.units = e->d_units; g.unit_cols = e->d_unit_cols; g.s_val = e->seg_copies ? e->d_unit_sval : e->d_sval; g.p_val = p_val;
    g.A = seg_rows_a(e); g.B = seg_rows_b(e);
    g.n_units = e->n_units;
    g.row_stride = static_cast<uint32_t>(e->Ks * elem_bytes(e));
    g.row_bytes = seg_row_bytes(e);
    g.one = 1.0f;
    if (int st = begin_kernel(e, stream)) return st;
    if (e->seg_slices > 1) {   // one launch per slice of K, in stream order
        g.row_bytes = 4 * e->slice_cols;
        if (e->slice_major) g.row_stride = 4 * e->slice_cols;
        for (int sl = 0; sl < e->seg_slices; ++sl) {
            const SliceStep step = sl == 0 ? kFirstSlice : sl + 1 < e->seg_slices ? kNextSlice : kLastSlice;
            CU_TRY(e, to.launch(side, pick_rowseg_slice(e, e->seg_copies, step), p.rowseg_grid, kRowSegWarps * 32, 0, g));
            g.A = static_cast<const float *>(g.A) + e->slice_cols * (e->slice_major ? e->M : 1);
            g.B = static_cast<const float *>(g.B) + e->slice_cols * (e->slice_major ? e->N : 1);
        }
    } else {
        CU_TRY(e, to.launch(side, seg_function(e, e->seg_copies), p.rowseg_grid, kRowSegWarps * 32, 0, g));
    }
    return mark_kernel(e, "sddmm_rowseg_kernel", stream);   // (the slices of one step count as one kernel in the timing table)
}

// every kernel of one run, P.val going to `p_val`
int launch_all(sddmm_b200_engine *e, float *p_val, cudaGraph_t graph = nullptr) {
    const sddmm_b200_plan_info &p = e->plan;
    RunTarget to{e, graph};
    e->kernels_launched = 0;
    if (e->nnz == 0) return SDDMM_B200_OK;
    int st = SDDMM_B200_OK;
    if (e->use_scalar && !e->use_seg) {
        if ((st = begin_kernel(e, e->stream))) return st;
        CU_TRY(e, to.launch(false, sddmm_scalar_kernel, p.rowtile_grid, kBlock, 0, e->d_rp, e->d_col, e->d_sval, p_val, e->d_A32, e->d_B32,
                            static_cast<int32_t>(e->M), static_cast<int32_t>(e->K), e->nnz));
        return mark_kernel(e, "sddmm_scalar_kernel", e->stream);
    }
    if (e->rg_rows && e->rg_units) {
        RowSegGroupArgs g;
        g.ghdr = reinterpret_cast<const int4 *>(e->d_units); g.unit_cols = e->d_unit_cols; g.s_val = e->d_sval; g.p_val = p_val;
        g.A = static_cast<const float *>(seg_rows_a(e)); g.B = static_cast<const float *>(seg_rows_b(e));
        g.n_units = e->n_units;
        g.row_bytes = static_cast<uint32_t>(e->Ks * elem_bytes(e));
        if ((st = begin_kernel(e, e->stream))) return st;
        CU_TRY(e, to.launch(false, pick_rowseg_group(e, e->rg_rows), p.rowgroup_grid, kRowSegWarps * 32, 0, g));
        return mark_kernel(e, "sddmm_rowseg_group_kernel", e->stream);
    }
    if (e->rg_rows) {
        RowGroupArgs g;
        g.row_ptr = e->d_rp; g.col_idx = e->d_col; g.s_val = e->d_sval; g.p_val = p_val; g.A = e->d_A32; g.B = e->d_B32;
        g.group_ok = e->d_group_ok; g.M = static_cast<int32_t>(e->M); g.K = static_cast<int32_t>(e->K); g.first = e->rg_first; g.n_groups = e->rg_groups;
        if ((st = begin_kernel(e, e->stream))) return st;
        CU_TRY(e, to.launch(false, pick_rowgroup(e->rg_rows, static_cast<int>(e->K / 32)), p.rowgroup_grid, kRowGroupWarps * 32, 0, g));
        return mark_kernel(e, "sddmm_rowgroup_kernel", e->stream);
    }
    if (e->use_seg && e->n_dense == 0) return launch_rowseg(e, to, false, p_val);
    // the two kernels write disjoint nonzeros: when both run, the row-tile kernel goes to the side stream
    static const bool no_side = std::getenv("SDDMM_B200_NO_SIDE_STREAM") != nullptr;   // tuning / debugging knob
    const bool both = e->n_dense > 0 && e->n_residual_items > 0 && !no_side;
    cudaStream_t rt_stream = both ? e->side_stream : e->stream;
    if (both && !graph) {   // (in a graph the two kernels are two nodes that do not depend on one another)
        CU_TRY(e, cudaEventRecord(e->ev_fork, e->stream));
        CU_TRY(e, cudaStreamWaitEvent(e->side_stream, e->ev_fork, 0));
    }
    if (e->n_dense > 0 && e->dense_fma) {
        DenseFmaArgs d;
        d.origins = e->dense_origin; d.descs = e->d_dense_descs; d.s_val = e->d_sval; d.p_val = p_val; d.A = e->d_A32; d.B = e->d_B32;
        d.n_tiles = e->n_dense; d.M = static_cast<int32_t>(e->M); d.N = static_cast<int32_t>(e->N); d.K = static_cast<int32_t>(e->K);
        if ((st = begin_kernel(e, e->stream))) return st;
        CU_TRY(e, to.launch(false, dense_fma_function(e->dense_own), p.dense_grid, kFmaThreads, 0, d));
        if ((st = mark_kernel(e, "sddmm_dense_tile_fma_kernel", e->stream))) return st;
        if (e->n_residual_items == 0) return SDDMM_B200_OK;
    } else if (e->n_dense > 0) {
        DenseArgs d;
        d.origins = e->dense_origin; d.descs = e->d_dense_descs; d.s_val = e->d_sval; d.p_val = p_val; d.err = e->h_err;
        d.n_tiles = e->n_dense;
        d.k_blocks = static_cast<int32_t>((e->mode == SDDMM_B200_FP32_TC ? 3 * e->K : e->K) / 32);
        d.nnz = e->nnz;
        if ((st = begin_kernel(e, e->stream))) return st;
        using DenseFn = void (*)(const DenseArgs, const CUtensorMap, const CUtensorMap);
        CU_TRY(e, to.launch(false, reinterpret_cast<DenseFn>(const_cast<void *>(dense_function(e->dense_own, e->dense_split3))), p.dense_grid, kDenseThreads,
                            p.dense_smem_bytes, d, e->map_a, e->map_b));
        if ((st = mark_kernel(e, "sddmm_dense_tile_kernel", e->stream))) return st;
        if (e->n_residual_items == 0) return SDDMM_B200_OK;
    }
    if (e->seg_residual) {
        if ((st = launch_rowseg(e, to, both, p_val))) return st;
        if (both && !graph) {
            CU_TRY(e, cudaEventRecord(e->ev_join, e->side_stream));
            CU_TRY(e, cudaStreamWaitEvent(e->stream, e->ev_join, 0));
        }
        return SDDMM_B200_OK;
    }
    RowTileArgs a;
    a.row_ptr = e->d_rp; a.col_idx = e->d_col; a.s_val = e->d_sval; a.p_val = p_val;
    a.item_rows = e->d_item_rows;
    a.item_ids = e->n_dense > 0 ? e->d_item_ids : nullptr;
    a.covered = e->n_dense > 0 ? e->d_covered : nullptr;
    a.err = e->h_err; a.nnz = e->nnz;
    a.M = static_cast<int32_t>(e->M); a.K = static_cast<int32_t>(e->K);   // (without row segments only, so that rows are K elements apart)
    a.n_items = p.rowtile_items; a.item_nnz = p.rowtile_item_nnz; a.rows_per_stage = p.rowtile_rows_per_stage;
    if ((st = begin_kernel(e, rt_stream))) return st;
    if (e->mode == SDDMM_B200_BF16) {
        a.A = e->d_A16; a.B = e->d_B16;
        CU_TRY(e, to.launch(both, pick_rowtile<__nv_bfloat16>(e->cpl, e->K == 32 * e->cpl), p.rowtile_grid, kBlock, p.rowtile_smem_bytes, a));
    } else {
        a.A = e->d_A32; a.B = e->d_B32;
        CU_TRY(e, to.launch(both, pick_rowtile<float>(e->cpl, e->K == 32 * e->cpl), p.rowtile_grid, kBlock, p.rowtile_smem_bytes, a));
    }
    if ((st = mark_kernel(e, "sddmm_rowtile_kernel", rt_stream))) return st;
    if (both && !graph) {
        CU_TRY(e, cudaEventRecord(e->ev_join, e->side_stream));
        CU_TRY(e, cudaStreamWaitEvent(e->stream, e->ev_join, 0));
    }
    return SDDMM_B200_OK;
}

// The plan's kernels as a graph (which holds their arguments: the engine's buffers stay where they are until the next upload).
int build_graph(sddmm_b200_engine *e) {
    cudaGraph_t g = nullptr;
    CU_TRY(e, cudaGraphCreate(&g, 0));
    int st = launch_all(e, e->d_pval, g);
    if (!st) st = cuda_status(e, cudaGraphInstantiate(&e->graph, g, 0));
    cudaGraphDestroy(g);
    if (st) e->graph = nullptr;
    return st;
}

// One run's kernels on the main stream.  The first runs of a plan launch them one by one (an upload per run pays for no
// graph); a later one builds their graph, which is replayed from then on.
int enqueue_run(sddmm_b200_engine *e) {
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    CU_TRY(e, cudaStreamIsCapturing(e->stream, &capturing));
    if (e->kernel_timing || e->nnz == 0 || capturing != cudaStreamCaptureStatusNone) return launch_all(e, e->d_pval);
    const bool specials = leave_out_past_end(e);
    if (e->graph && e->graph_specials != specials) drop_graph(e);   // (new values of B want the other kernels)
    if (!e->graph && e->runs_of_plan <= sddmm_b200_engine::kGraphAfter && ++e->runs_of_plan > sddmm_b200_engine::kGraphAfter) {
        if (build_graph(e) != SDDMM_B200_OK) cudaGetLastError();   // (no memory for one, say: this plan goes on without)
        e->graph_specials = specials;
    }
    if (!e->graph) return launch_all(e, e->d_pval);
    CU_TRY(e, cudaGraphLaunch(e->graph, e->stream));
    return SDDMM_B200_OK;
}

// B = NULL in an upload: take the B that sddmm_b200_stage_b left on this engine's device (same N and K)
int take_staged_b(sddmm_b200_engine *e, int64_t N, int64_t K, const float *B) {
    if (B) return SDDMM_B200_OK;
    if (!e->b_stage || e->b_stage_n != N || e->b_stage_k != K)
        return fail(e, SDDMM_B200_ERR_ARG, "B = NULL needs a B of the same shape staged by sddmm_b200_stage_b");
    if (!e->B_on_device) e->B_on_device = e->b_stage;   // (a chunked call sets its own source)
    return SDDMM_B200_OK;
}

}  // namespace

extern "C" {

const char *sddmm_b200_version(void) { return "sddmm_b200 0.1 (sm_100a)"; }

int sddmm_b200_device_count(void) {
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

int sddmm_b200_create(sddmm_b200_engine **out, int device, int mode, uint32_t flags) {
    if (!out) return SDDMM_B200_ERR_ARG;
    *out = nullptr;
    if (mode < SDDMM_B200_FP32 || mode > SDDMM_B200_FP32_TC) return SDDMM_B200_ERR_ARG;
    int n = sddmm_b200_device_count();
    if (n <= 0 || device < 0 || device >= n) return SDDMM_B200_ERR_CUDA;
    sddmm_b200_engine *e = new (std::nothrow) sddmm_b200_engine();
    if (!e) return SDDMM_B200_ERR_OOM;
    e->device = device;
    e->mode = mode;
    e->flags = flags;
    e->knob_panels = env_double("SDDMM_B200_PANELS", -1);
    e->knob_panel_mb = env_double("SDDMM_B200_PANEL_MB", -1);
    e->knob_rowseg = env_double("SDDMM_B200_ROWSEG", -1);
    e->knob_group_units = env_double("SDDMM_B200_GROUP_UNITS", -1);
    e->knob_offset_tiles = env_double("SDDMM_B200_OFFSET_TILES", -1);
    e->knob_dense_split3 = env_double("SDDMM_B200_DENSE_SPLIT3", -1);
    e->knob_k_slices = env_double("SDDMM_B200_K_SLICES", -1);
    e->knob_long_rows = env_double("SDDMM_B200_LONG_ROWS", -1);
    DeviceGuard g(device);
    DevicePool::instance().add_user(device);
    PinnedPool::instance().add_user();
    bool ok = g.ok;
    ok = ok && cudaStreamCreateWithFlags(&e->stream, cudaStreamNonBlocking) == cudaSuccess;
    ok = ok && cudaStreamCreateWithFlags(&e->side_stream, cudaStreamNonBlocking) == cudaSuccess;
    for (int i = 0; i < sddmm_b200_engine::kMaxKernels; ++i)
        ok = ok && cudaEventCreate(&e->ev_begin[i]) == cudaSuccess && cudaEventCreate(&e->ev_end[i]) == cudaSuccess;
    ok = ok && cudaEventCreate(&e->ev_run0) == cudaSuccess && cudaEventCreate(&e->ev_run1) == cudaSuccess;
    ok = ok && cudaEventCreate(&e->ev_spmm0) == cudaSuccess && cudaEventCreate(&e->ev_spmm1) == cudaSuccess;
    for (cudaEvent_t &ev : e->ev_chunk) ok = ok && cudaEventCreateWithFlags(&ev, cudaEventDisableTiming) == cudaSuccess;
    ok = ok && cudaEventCreateWithFlags(&e->ev_stage, cudaEventDisableTiming) == cudaSuccess;
    ok = ok && cudaEventCreateWithFlags(&e->ev_fork, cudaEventDisableTiming) == cudaSuccess;
    ok = ok && cudaEventCreateWithFlags(&e->ev_join, cudaEventDisableTiming) == cudaSuccess;
    ok = ok && cudaEventCreateWithFlags(&e->ev_h2d, cudaEventDisableTiming) == cudaSuccess;
    ok = ok && cudaDeviceGetAttribute(&e->sm_count, cudaDevAttrMultiProcessorCount, device) == cudaSuccess;
    ok = ok && cudaDeviceGetAttribute(&e->l2_bytes, cudaDevAttrL2CacheSize, device) == cudaSuccess;
    ok = ok && cudaHostAlloc(reinterpret_cast<void **>(&e->h_err), 2 * sizeof(int32_t), cudaHostAllocDefault) == cudaSuccess;
    ok = ok && cudaHostAlloc(reinterpret_cast<void **>(&e->h_pc), sizeof(PlanCounters), cudaHostAllocDefault) == cudaSuccess;
    if (!ok) {
        cudaGetLastError();
        sddmm_b200_destroy(e);
        return SDDMM_B200_ERR_CUDA;
    }
    *e->h_err = 0;
    e->h_specials = e->h_err + 1;
    *out = e;
    return SDDMM_B200_OK;
}

int sddmm_b200_destroy(sddmm_b200_engine *e) {
    if (!e) return SDDMM_B200_OK;
    {
        DeviceGuard g(e->device);
        if (e->stream) cudaStreamSynchronize(e->stream);
        if (e->side_stream) cudaStreamSynchronize(e->side_stream);
        drop_graph(e);
        e->arena.release(e->device);
        e->spmm_arena.release(e->device);
        e->b_stage_arena.release(e->device);
        DevicePool::instance().remove_user(e->device);
        e->stager.release();
        e->stager2.release();
        PinnedPool::instance().remove_user();
        if (e->ev_stage) cudaEventDestroy(e->ev_stage);
        if (e->ev_spmm0) cudaEventDestroy(e->ev_spmm0);
        if (e->ev_spmm1) cudaEventDestroy(e->ev_spmm1);
        for (cudaEvent_t ev : e->ev_chunk)
            if (ev) cudaEventDestroy(ev);
        if (e->h_err) cudaFreeHost(e->h_err);
        if (e->h_pc) cudaFreeHost(e->h_pc);
        for (int i = 0; i < sddmm_b200_engine::kMaxKernels; ++i) {
            if (e->ev_begin[i]) cudaEventDestroy(e->ev_begin[i]);
            if (e->ev_end[i]) cudaEventDestroy(e->ev_end[i]);
        }
        for (cudaEvent_t ev : {e->ev_run0, e->ev_run1, e->ev_fork, e->ev_join, e->ev_h2d})
            if (ev) cudaEventDestroy(ev);
        if (e->side_stream) cudaStreamDestroy(e->side_stream);
        if (e->stream) cudaStreamDestroy(e->stream);
    }
    delete e;
    return SDDMM_B200_OK;
}

int sddmm_b200_upload_csr(sddmm_b200_engine *e, int64_t M, int64_t N, int64_t K, const int32_t *row_ptr,
                          const int32_t *col_idx, const float *s_val, const float *A, const float *B) {
    if (!e) return SDDMM_B200_ERR_ARG;
    if (!row_ptr || !A) return fail(e, SDDMM_B200_ERR_ARG, "null pointer argument");
    if (M < 1) return fail(e, SDDMM_B200_ERR_ARG, "need M >= 1");
    const int64_t nnz = row_ptr[M];
    int st = check_dims(e, M, N, K, nnz);
    if (st) return st;
    if (nnz > 0 && (!col_idx || !s_val)) return fail(e, SDDMM_B200_ERR_ARG, "null pointer argument");
    if ((st = take_staged_b(e, N, K, B))) return st;
    DeviceGuard g(e->device);
    return upload_common(e, M, N, K, nnz, row_ptr, nullptr, col_idx, s_val, A, B, cudaMemcpyHostToDevice);
}

int sddmm_b200_upload_coo(sddmm_b200_engine *e, int64_t M, int64_t N, int64_t K, int64_t nnz, const int32_t *row_idx,
                          const int32_t *col_idx, const float *s_val, const float *A, const float *B) {
    if (!e) return SDDMM_B200_ERR_ARG;
    if (!A) return fail(e, SDDMM_B200_ERR_ARG, "null pointer argument");
    int st = check_dims(e, M, N, K, nnz);
    if (st) return st;
    if (nnz > 0 && (!row_idx || !col_idx || !s_val)) return fail(e, SDDMM_B200_ERR_ARG, "null pointer argument");
    if ((st = take_staged_b(e, N, K, B))) return st;
    DeviceGuard g(e->device);
    static const int32_t dummy = 0;
    return upload_common(e, M, N, K, nnz, nullptr, nnz ? row_idx : &dummy, col_idx, s_val, A, B, cudaMemcpyHostToDevice);
}

int sddmm_b200_upload_coo_rows(sddmm_b200_engine *e, int64_t M, int64_t N, int64_t K, int64_t nnz, int64_t row_base, const int32_t *row_idx,
                               const int32_t *col_idx, const float *s_val, const float *A, const float *B) {
    if (!e) return SDDMM_B200_ERR_ARG;
    if (row_base < 0 || row_base + M >= (int64_t(1) << 31)) return fail(e, SDDMM_B200_ERR_ARG, "row_base outside the int32 index range");
    e->coo_row_base = static_cast<int32_t>(row_base);
    const int st = sddmm_b200_upload_coo(e, M, N, K, nnz, row_idx, col_idx, s_val, A, B);
    e->coo_row_base = 0;
    return st;
}

int sddmm_b200_upload_csr_device(sddmm_b200_engine *e, int64_t M, int64_t N, int64_t K, const int32_t *row_ptr,
                                 const int32_t *col_idx, const float *s_val, const float *A, const float *B) {
    if (!e) return SDDMM_B200_ERR_ARG;
    if (!row_ptr || !A || !B) return fail(e, SDDMM_B200_ERR_ARG, "null pointer argument");
    if (M < 1) return fail(e, SDDMM_B200_ERR_ARG, "need M >= 1");
    DeviceGuard g(e->device);
    int32_t last = 0;
    // (on the legacy stream, as a plain cudaMemcpy: behind what the caller has enqueued there; into pinned memory, which saves a staged copy)
    CU_TRY(e, cudaMemcpyAsync(e->h_pc, row_ptr + M, sizeof(int32_t), cudaMemcpyDeviceToHost, cudaStreamLegacy));
    CU_TRY(e, cudaStreamSynchronize(cudaStreamLegacy));
    std::memcpy(&last, e->h_pc, sizeof(int32_t));
    const int64_t nnz = last;
    int st = check_dims(e, M, N, K, nnz);
    if (st) return st;
    if (nnz > 0 && (!col_idx || !s_val)) return fail(e, SDDMM_B200_ERR_ARG, "null pointer argument");
    return upload_common(e, M, N, K, nnz, row_ptr, nullptr, col_idx, s_val, A, B, cudaMemcpyDeviceToDevice);
}

int sddmm_b200_update_dense(sddmm_b200_engine *e, const float *A, const float *B) {
    if (!e) return SDDMM_B200_ERR_ARG;
    if (!e->uploaded) return fail(e, SDDMM_B200_ERR_STATE, "update_dense before upload");
    DeviceGuard g(e->device);
    if (A) CU_TRY(e, e->stager.upload(e->d_A32, A, static_cast<size_t>(e->M * e->K) * 4, e->stream));
    if (B) CU_TRY(e, e->stager.upload(e->d_B32, B, static_cast<size_t>(e->N * e->K) * 4, e->stream));
    int st = convert_storage(e);
    if (st) return st;
    CU_TRY(e, cudaStreamSynchronize(e->stream));
    settle_specials(e);
    return SDDMM_B200_OK;
}

int sddmm_b200_update_values(sddmm_b200_engine *e, const float *s_val) {
    if (!e) return SDDMM_B200_ERR_ARG;
    if (!e->uploaded) return fail(e, SDDMM_B200_ERR_STATE, "update_values before upload");
    if (!s_val && e->nnz) return fail(e, SDDMM_B200_ERR_ARG, "null pointer argument");
    DeviceGuard g(e->device);
    if (e->nnz) CU_TRY(e, e->stager.upload(e->d_sval, s_val, static_cast<size_t>(e->nnz) * 4, e->stream));
    if (int rc = refresh_unit_values(e)) return rc;
    CU_TRY(e, cudaStreamSynchronize(e->stream));
    return SDDMM_B200_OK;
}

int sddmm_b200_run(sddmm_b200_engine *e) {
    if (!e) return SDDMM_B200_ERR_ARG;
    if (!e->uploaded) return fail(e, SDDMM_B200_ERR_STATE, "run before upload");
    DeviceGuard g(e->device);
    // (a wait that ran out in an earlier run must not be reported again: the error word starts every run clean)
    *static_cast<volatile int32_t *>(e->h_err) = kDevOk;
    e->last_run_timed = e->kernel_timing;
    const bool timed = e->run_timing || e->kernel_timing;
    if (timed) CU_TRY(e, cudaEventRecord(e->ev_run0, e->stream));
    int st = enqueue_run(e);
    if (st) return st;
    if (timed) CU_TRY(e, cudaEventRecord(e->ev_run1, e->stream));
    e->last_run_timed_whole = timed;
    e->ran = true;
    return SDDMM_B200_OK;
}

int sddmm_b200_sync(sddmm_b200_engine *e) {
    if (!e) return SDDMM_B200_ERR_ARG;
    DeviceGuard g(e->device);
    CU_TRY(e, cudaStreamSynchronize(e->stream));
    const int32_t code = *static_cast<volatile int32_t *>(e->h_err);
    if (e->ran && code != kDevOk) return fail(e, SDDMM_B200_ERR_DEVICE_WAIT, "device-side bounded wait ran out (code %d)", code);
    return SDDMM_B200_OK;
}

int sddmm_b200_download(sddmm_b200_engine *e, float *p_val) {
    if (!e) return SDDMM_B200_ERR_ARG;
    if (!e->uploaded || !e->ran) return fail(e, SDDMM_B200_ERR_STATE, "download before run");
    if (!p_val && e->nnz) return fail(e, SDDMM_B200_ERR_ARG, "null pointer argument");
    DeviceGuard g(e->device);
    if (e->nnz) CU_TRY(e, e->stager.download(p_val, e->d_pval, static_cast<size_t>(e->nnz) * 4, e->stream));
    return sddmm_b200_sync(e);
}

int sddmm_b200_p_device(sddmm_b200_engine *e, float **p) {
    if (!e || !p) return SDDMM_B200_ERR_ARG;
    if (!e->uploaded) return fail(e, SDDMM_B200_ERR_STATE, "p_device before upload");
    e->arena.exposed = true;
    *p = e->d_pval;
    return SDDMM_B200_OK;
}

int sddmm_b200_last_run_ms(sddmm_b200_engine *e, float *ms) {
    if (!e || !ms) return SDDMM_B200_ERR_ARG;
    e->run_timing = true;   // every later run() records the pair
    if (!e->ran) return fail(e, SDDMM_B200_ERR_STATE, "last_run_ms before run");
    DeviceGuard g(e->device);
    *ms = 0.f;
    if (e->kernels_launched == 0) return SDDMM_B200_OK;
    if (!e->last_run_timed_whole) {
        // nobody had asked for run times yet, so the last run recorded no events: its kernels are launched once more between two,
        // into a buffer of their own -- P.val and whatever the caller has done with it stay.  Where the device has no room for one,
        // P.val is put aside in host memory meanwhile.
        const size_t bytes = static_cast<size_t>(e->nnz) * 4;
        size_t cap = 0;
        float *scratch = static_cast<float *>(DevicePool::instance().take(e->device, bytes + 16, &cap));
        std::unique_ptr<char[]> aside;
        cudaError_t err = cudaSuccess;
        if (!scratch) {
            aside.reset(new (std::nothrow) char[bytes]);
            if (!aside) return fail(e, SDDMM_B200_ERR_OOM, "%zu bytes to repeat the run for its time", bytes);
            err = cudaMemcpyAsync(aside.get(), e->d_pval, bytes, cudaMemcpyDeviceToHost, e->stream);
            if (err == cudaSuccess) err = cudaStreamSynchronize(e->stream);
            if (err != cudaSuccess) return cuda_status(e, err);
        }
        int st = cuda_status(e, cudaEventRecord(e->ev_run0, e->stream));
        if (!st) st = launch_all(e, scratch ? scratch : e->d_pval);
        if (!st) st = cuda_status(e, cudaEventRecord(e->ev_run1, e->stream));
        if (aside) err = cudaMemcpyAsync(e->d_pval, aside.get(), bytes, cudaMemcpyHostToDevice, e->stream);
        const cudaError_t drained = cudaStreamSynchronize(e->stream);
        DevicePool::instance().put(e->device, scratch, cap);
        if (st) return st;
        CU_TRY(e, err);
        CU_TRY(e, drained);
        e->last_run_timed_whole = true;
    }
    CU_TRY(e, cudaEventSynchronize(e->ev_run1));
    CU_TRY(e, cudaEventElapsedTime(ms, e->ev_run0, e->ev_run1));
    return SDDMM_B200_OK;
}

int sddmm_b200_last_kernel_ms(sddmm_b200_engine *e, int index, float *ms, const char **name) {
    if (!e || !ms) return SDDMM_B200_ERR_ARG;
    if (!e->ran) return fail(e, SDDMM_B200_ERR_STATE, "last_kernel_ms before run");
    if (index < 0 || index >= e->kernels_launched) return fail(e, SDDMM_B200_ERR_ARG, "kernel index %d of %d", index, e->kernels_launched);
    if (name) *name = e->kernel_name[index];
    if (!e->last_run_timed) {   // names are always known, times only when the run was asked to record them
        *ms = -1.f;
        return SDDMM_B200_OK;
    }
    DeviceGuard g(e->device);
    CU_TRY(e, cudaEventSynchronize(e->ev_end[index]));
    CU_TRY(e, cudaEventElapsedTime(ms, e->ev_begin[index], e->ev_end[index]));
    return SDDMM_B200_OK;
}

int sddmm_b200_set_kernel_timing(sddmm_b200_engine *e, int enabled) {
    if (!e) return SDDMM_B200_ERR_ARG;
    e->kernel_timing = enabled != 0;
    return SDDMM_B200_OK;
}

// ---- self-test of the bounded device-side wait --------------------------------------------------------------
namespace {
// One thread waits, with the given probe limit, on an mbarrier phase that nothing ever completes, records the time-out
// in the error word exactly as the kernels do, and returns.  Nothing faults and nothing hangs: the wait is bounded.
__global__ void k_wait_timeout_selftest(int32_t *err, uint32_t limit) {
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x == 0) {
        mbar_init(&bar, 1);
        fence_mbar_init();
        if (!mbar_wait_bounded(&bar, 0u, limit)) record_error(err, kDevMbarrierTimeout);
    }
}
}  // namespace

int sddmm_b200_selftest_wait_timeout(sddmm_b200_engine *e, int probes) {
    if (!e) return SDDMM_B200_ERR_ARG;
    if (!e->uploaded) return fail(e, SDDMM_B200_ERR_STATE, "selftest before upload (the error word lives in the upload's buffers)");
    if (probes < 1 || probes > (1 << 16)) return fail(e, SDDMM_B200_ERR_ARG, "probes must be in [1, 65536]");
    DeviceGuard g(e->device);
    *static_cast<volatile int32_t *>(e->h_err) = kDevOk;
    k_wait_timeout_selftest<<<1, 32, 0, e->stream>>>(e->h_err, static_cast<uint32_t>(probes));
    CU_TRY(e, cudaGetLastError());
    e->ran = true;   // sync() reports the error word of the last enqueued work
    return sddmm_b200_sync(e);
}

int sddmm_b200_row_cuts(const int32_t *row_ptr, int64_t M, int parts, int64_t align, int64_t *cuts) {
    if (!row_ptr || !cuts || M < 0 || parts < 1) return SDDMM_B200_ERR_ARG;
    const int64_t nnz = row_ptr[M];
    cuts[0] = 0;
    cuts[parts] = M;
    for (int g = 1; g < parts; ++g) {
        const int64_t target = nnz * g / parts;
        int64_t r = std::lower_bound(row_ptr, row_ptr + M + 1, target) - row_ptr;   // first boundary at or past the target
        r = std::min<int64_t>(r, M);
        if (r > 0 && target - row_ptr[r - 1] < row_ptr[r] - target) --r;              // the closer boundary wins
        if (align > 1) r = (r + align / 2) / align * align;
        cuts[g] = std::max<int64_t>(cuts[g - 1], std::min<int64_t>(r, M));
    }
    return SDDMM_B200_OK;
}

int sddmm_b200_coo_cuts(const int32_t *row_idx, int64_t nnz, int64_t M, int parts, int64_t align, int64_t *cuts, int64_t *offsets) {
    if (!cuts || !offsets || M < 0 || nnz < 0 || parts < 1 || (nnz > 0 && !row_idx)) return SDDMM_B200_ERR_ARG;
    cuts[0] = 0;
    offsets[0] = 0;
    cuts[parts] = M;
    offsets[parts] = nnz;
    for (int g = 1; g < parts; ++g) {
        int64_t r = nnz ? row_idx[std::min<int64_t>(nnz - 1, nnz * g / parts)] : 0;   // the row holding the part's first nonzero ...
        if (r < 0 || r >= std::max<int64_t>(M, 1)) return SDDMM_B200_ERR_INDEX;
        if (align > 1) r = std::min<int64_t>((r + align / 2) / align * align, M);
        r = std::max<int64_t>(r, cuts[g - 1]);
        const int64_t pos = std::lower_bound(row_idx, row_idx + nnz, static_cast<int32_t>(r)) - row_idx;   // ... taken whole
        cuts[g] = r;
        offsets[g] = std::max<int64_t>(pos, offsets[g - 1]);
    }
    for (int g = 0; g < parts; ++g)   // nonzeros in a part without rows: the rows cannot be sorted
        if (cuts[g + 1] == cuts[g] && offsets[g + 1] != offsets[g]) return SDDMM_B200_ERR_INDEX;
    return SDDMM_B200_OK;
}

int sddmm_b200_stage_b(sddmm_b200_engine **engines, int n, int64_t N, int64_t K, const float *B) {
    if (!engines || n < 1 || !B || N < 1 || K < 1) return SDDMM_B200_ERR_ARG;
    for (int i = 0; i < n; ++i)
        if (!engines[i]) return SDDMM_B200_ERR_ARG;
    const size_t bytes = static_cast<size_t>(N) * static_cast<size_t>(K) * 4;
    // a staging buffer on every engine's device
    for (int i = 0; i < n; ++i) {
        sddmm_b200_engine *e = engines[i];
        DeviceGuard g(e->device);
        if (!g.ok) return fail(e, SDDMM_B200_ERR_COMM, "device %d cannot be selected", e->device);
        e->b_stage_n = e->b_stage_k = 0;
        if (e->b_stage_arena.cap < bytes) {   // (from the pool, which gives its buffers back when memory is short)
            e->b_stage = nullptr;
            if (cudaStreamSynchronize(e->stream) != cudaSuccess || cudaStreamSynchronize(e->side_stream) != cudaSuccess) {
                cudaGetLastError();
                return fail(e, SDDMM_B200_ERR_CUDA, "device %d: earlier work failed", e->device);
            }
            if (!e->b_stage_arena.grow(e->device, bytes))
                return fail(e, SDDMM_B200_ERR_OOM, "staging buffer for B (%zu bytes) on device %d", bytes, e->device);
            e->b_stage = reinterpret_cast<float *>(e->b_stage_arena.base);
        }
    }
    // the host link is crossed once; then the copy doubles the set of devices that hold B in every round
    // (device to device: over NVLink where the devices are peers, through the host otherwise)
    int rc = SDDMM_B200_OK;
    {
        sddmm_b200_engine *e0 = engines[0];
        DeviceGuard g(e0->device);
        if (e0->stager.upload(e0->b_stage, B, bytes, e0->stream) != cudaSuccess ||
            cudaEventRecord(e0->ev_stage, e0->stream) != cudaSuccess)
            rc = fail(e0, SDDMM_B200_ERR_COMM, "upload of B to device %d: %s", e0->device, cudaGetErrorString(cudaGetLastError()));
    }
    for (int have = 1; have < n && !rc; have *= 2) {
        for (int i = 0; i < have && have + i < n && !rc; ++i) {
            sddmm_b200_engine *src = engines[i], *dst = engines[have + i];
            DeviceGuard g(dst->device);
            cudaError_t st = cudaStreamWaitEvent(dst->stream, src->ev_stage, 0);
            if (st == cudaSuccess) {
                if (src->device == dst->device) {
                    st = cudaMemcpyAsync(dst->b_stage, src->b_stage, bytes, cudaMemcpyDeviceToDevice, dst->stream);
                } else {
                    int can = 0;
                    if (cudaDeviceCanAccessPeer(&can, dst->device, src->device) == cudaSuccess && can) {
                        const cudaError_t pe = cudaDeviceEnablePeerAccess(src->device, 0);   // (already enabled is fine)
                        if (pe != cudaSuccess) cudaGetLastError();
                    }
                    st = cudaMemcpyPeerAsync(dst->b_stage, dst->device, src->b_stage, src->device, bytes, dst->stream);
                }
            }
            if (st == cudaSuccess) st = cudaEventRecord(dst->ev_stage, dst->stream);
            if (st != cudaSuccess) {
                cudaGetLastError();
                rc = fail(dst, SDDMM_B200_ERR_COMM, "copy of B from device %d to device %d: %s", src->device, dst->device, cudaGetErrorString(st));
            }
        }
    }
    for (int i = 0; i < n; ++i) {   // drain every stream, also after a failure: nothing may still read the caller's buffer
        sddmm_b200_engine *e = engines[i];
        DeviceGuard g(e->device);
        if (cudaStreamSynchronize(e->stream) != cudaSuccess && !rc) {
            cudaGetLastError();
            rc = fail(e, SDDMM_B200_ERR_COMM, "copy of B to device %d did not complete", e->device);
        }
    }
    if (rc) return rc;
    for (int i = 0; i < n; ++i) {
        engines[i]->b_stage_n = N;
        engines[i]->b_stage_k = K;
    }
    return SDDMM_B200_OK;
}

int sddmm_b200_set_knob(sddmm_b200_engine *e, const char *name, double value) {
    if (!e || !name) return SDDMM_B200_ERR_ARG;
    struct { const char *name; double *slot; } knobs[] = {
        {"panels", &e->knob_panels}, {"panel_mb", &e->knob_panel_mb}, {"rowseg", &e->knob_rowseg},
        {"b_fraction", nullptr}, {"group_units", &e->knob_group_units},
        {"offset_tiles", &e->knob_offset_tiles}, {"dense_split3", &e->knob_dense_split3}, {"k_slices", &e->knob_k_slices}, {"long_rows", &e->knob_long_rows},
    };
    for (auto &k : knobs)
        if (std::strcmp(name, k.name) == 0) {
            if (k.slot) *k.slot = value;   // (accepted, without effect)
            drop_graph(e);
            return SDDMM_B200_OK;
        }
    return fail(e, SDDMM_B200_ERR_ARG, "unknown knob '%s'", name);
}

// ---- consumer of P on the device: Y = P X ----------------------------------------------------------------
namespace {
using SpmmFn = void (*)(const SpmmArgs);
SpmmFn pick_spmm(int cpl, bool exact) {
    switch (cpl) {
        case 1: return exact ? sddmm_spmm_kernel<1, true> : sddmm_spmm_kernel<1, false>;
        case 2: return exact ? sddmm_spmm_kernel<2, true> : sddmm_spmm_kernel<2, false>;
        case 4: return exact ? sddmm_spmm_kernel<4, true> : sddmm_spmm_kernel<4, false>;
        case 8: return exact ? sddmm_spmm_kernel<8, true> : sddmm_spmm_kernel<8, false>;
        default: return nullptr;
    }
}

// X (unless it is B), Y and the consumer's unit list live in their own buffer (grown on demand, kept across calls).  Where
// the run itself works on whole rows its list is the consumer's too.
int spmm_prepare(sddmm_b200_engine *e, int64_t K2, bool own_x) {
    Carve c;
    const size_t M = static_cast<size_t>(e->M), N = static_cast<size_t>(e->N), nnz = static_cast<size_t>(e->nnz);
    const size_t cap = nnz / 8 + std::min(M, nnz) + 8;
    const bool shared = e->use_seg && e->n_dense == 0 && !e->rg_rows && e->plan.rowseg_panels == 1 && e->n_units > 0;
    const size_t o_u = shared ? 0 : c.take(cap * sizeof(int2)), o_y = c.take(M * K2 * 4), o_x = own_x ? c.take(N * K2 * 4) : 0;
    if (int rc = grow_arena(e, e->spmm_arena, c.off, "consumer buffers")) return rc;
    char *b = e->spmm_arena.base;
    e->d_X = own_x ? reinterpret_cast<float *>(b + o_x) : nullptr;
    e->d_Y = reinterpret_cast<float *>(b + o_y);
    e->d_spmm_units = shared ? e->d_units : reinterpret_cast<int2 *>(b + o_u);
    e->spmm_k2 = K2;
    if (!shared && e->spmm_list_in != e->spmm_arena.buffers) e->spmm_units = 0;   // the list went with the buffer it was in
    e->spmm_list_in = e->spmm_arena.buffers;
    if (e->spmm_units == 0 && shared) {
        k_unit_cuts<<<1, 32, 0, e->stream>>>(e->d_units, static_cast<int32_t>(e->M), sddmm_b200_engine::kSpmmChunks, e->n_units, e->d_pc);
        CU_TRY(e, cudaGetLastError());
        PlanCounters pc;
        if (int rc = read_counters(e, &pc)) return rc;
        e->spmm_units = e->n_units;
        for (int k = 1; k < sddmm_b200_engine::kSpmmChunks; ++k) e->spmm_cut[k] = pc.unit_cut[k];
    } else if (e->spmm_units == 0) {   // plain row segments (one panel, no groups), counted / scanned / written on the device
        const int32_t Mi = static_cast<int32_t>(e->M);
        cudaStream_t s = e->stream;
        const RunsOfRows runs{e->d_rp, e->d_col, Mi, static_cast<int32_t>(e->nnz)};
        if (int rc = enqueue_units(e, s, runs, e->M, false, static_cast<int64_t>(cap), e->d_spmm_units, static_cast<int32_t *>(nullptr))) return rc;
        k_unit_cuts<<<1, 32, 0, s>>>(e->d_spmm_units, Mi, sddmm_b200_engine::kSpmmChunks, -1, e->d_pc);
        CU_TRY(e, cudaGetLastError());
        PlanCounters pc;
        if (int rc = read_counters(e, &pc)) return rc;
        if (pc.units == 0 || pc.units > cap) return fail(e, SDDMM_B200_ERR_CUDA, "consumer plan: %llu units for a list of %zu", pc.units, cap);
        e->spmm_units = static_cast<int32_t>(pc.units);
        for (int c = 1; c < sddmm_b200_engine::kSpmmChunks; ++c) e->spmm_cut[c] = pc.unit_cut[c];
    }
    e->spmm_cut[0] = 0;
    e->spmm_cut[sddmm_b200_engine::kSpmmChunks] = e->spmm_units;
    return SDDMM_B200_OK;
}
}  // namespace

int sddmm_b200_spmm(sddmm_b200_engine *e, int64_t K2, const float *X, float *Y) {
    if (!e) return SDDMM_B200_ERR_ARG;
    if (!e->uploaded || !e->ran) return fail(e, SDDMM_B200_ERR_STATE, "spmm before run");
    if (K2 < 4 || K2 % 4 != 0 || K2 > 256) return fail(e, SDDMM_B200_ERR_UNSUPPORTED, "the consumer needs K2 %% 4 == 0 and 4 <= K2 <= 256 (K2 = %lld)", (long long)K2);
    if (!Y) return fail(e, SDDMM_B200_ERR_ARG, "null pointer argument");
    if (!X && K2 != e->K) return fail(e, SDDMM_B200_ERR_ARG, "X = NULL means X = B, which needs K2 == K");
    if (e->M >= kUnitRowLimit) return fail(e, SDDMM_B200_ERR_UNSUPPORTED, "the consumer handles fewer than 2^28 rows");
    DeviceGuard g(e->device);
    cudaStream_t s = e->stream;
    const size_t ybytes = static_cast<size_t>(e->M) * K2 * 4;
    if (e->nnz == 0) {
        std::memset(Y, 0, ybytes);
        return sddmm_b200_sync(e);
    }
    int st = spmm_prepare(e, K2, X != nullptr);   // (uses the plan scratch of the main arena: nothing of the run still needs it)
    if (st) return st;
    if (X) CU_TRY(e, cudaMemcpyAsync(e->d_X, X, static_cast<size_t>(e->N) * K2 * 4, cudaMemcpyHostToDevice, s));
    CU_TRY(e, cudaEventRecord(e->ev_spmm0, s));
    CU_TRY(e, cudaMemsetAsync(e->d_Y, 0, ybytes, s));
    const int cpl = round_up_cpl(K2);
    SpmmFn fn = pick_spmm(cpl, K2 == 32 * cpl);
    int occ = 0;
    CU_TRY(e, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, fn, kSpmmWarps * 32, 0));
    if (occ < 1) return fail(e, SDDMM_B200_ERR_CUDA, "consumer kernel does not fit on an SM");
    // Row ranges of about 4 MB of Y: while a range crosses the link the next one is computed (the copy of all of Y after the
    // whole kernel: 100 003 rows, K2 = 64, 103 us of kernel before 465 us of copy).
    constexpr int kMost = sddmm_b200_engine::kSpmmChunks;
    const int chunks = ybytes >= (size_t(32) << 20) ? 8 : ybytes >= (size_t(16) << 20) ? 4 : ybytes >= (size_t(8) << 20) ? 2 : 1;
    int64_t row[kMost + 1];
    for (int c = 0; c <= chunks; ++c) row[c] = range_start(e->M, c * (kMost / chunks), kMost);
    for (int c = 0; c < chunks; ++c) {
        const int32_t u0 = e->spmm_cut[c * (kMost / chunks)], u1 = e->spmm_cut[(c + 1) * (kMost / chunks)];
        if (u1 > u0) {
            SpmmArgs a;
            a.units = e->d_spmm_units + u0; a.col_idx = e->d_col; a.p_val = e->d_pval; a.X = X ? e->d_X : e->d_B32; a.Y = e->d_Y;
            a.n_units = u1 - u0; a.K2 = static_cast<int32_t>(K2);
            const int64_t n_quads = (static_cast<int64_t>(a.n_units) + 3) / 4;
            const int grid = static_cast<int>(std::min<int64_t>((n_quads + kSpmmWarps - 1) / kSpmmWarps, static_cast<int64_t>(e->sm_count) * occ));
            fn<<<grid, kSpmmWarps * 32, 0, s>>>(a);
            CU_TRY(e, cudaGetLastError());
        }
        CU_TRY(e, cudaEventRecord(e->ev_chunk[c], s));
    }
    CU_TRY(e, cudaEventRecord(e->ev_spmm1, s));
    for (int c = 0; c < chunks; ++c) {
        CU_TRY(e, cudaStreamWaitEvent(e->side_stream, e->ev_chunk[c], 0));
        const size_t at = static_cast<size_t>(row[c]) * K2, n = static_cast<size_t>(row[c + 1] - row[c]) * K2;
        if (n) CU_TRY(e, e->stager2.download(Y + at, e->d_Y + at, n * 4, e->side_stream));
    }
    CU_TRY(e, cudaStreamSynchronize(e->side_stream));
    return sddmm_b200_sync(e);
}

int sddmm_b200_last_spmm_ms(sddmm_b200_engine *e, float *ms) {
    if (!e || !ms) return SDDMM_B200_ERR_ARG;
    if (!e->spmm_k2) return fail(e, SDDMM_B200_ERR_STATE, "last_spmm_ms before spmm");
    DeviceGuard g(e->device);
    CU_TRY(e, cudaEventSynchronize(e->ev_spmm1));
    CU_TRY(e, cudaEventElapsedTime(ms, e->ev_spmm0, e->ev_spmm1));
    return SDDMM_B200_OK;
}

int sddmm_b200_get_plan(sddmm_b200_engine *e, sddmm_b200_plan_info *info) {
    if (!e || !info) return SDDMM_B200_ERR_ARG;
    if (!e->uploaded) return fail(e, SDDMM_B200_ERR_STATE, "get_plan before upload");
    *info = e->plan;
    return SDDMM_B200_OK;
}

int64_t sddmm_b200_algorithmic_bytes(sddmm_b200_engine *e) {
    if (!e || !e->uploaded) return -1;
    const int64_t eb = static_cast<int64_t>(elem_bytes(e));
    return eb * e->K * (e->plan.rows_nonempty + e->plan.cols_touched) + 12 * e->nnz + 4 * (e->M + 1);
}

int64_t sddmm_b200_flops(sddmm_b200_engine *e) {
    if (!e || !e->uploaded) return -1;
    return 2 * e->nnz * e->K;
}

const char *sddmm_b200_last_error(sddmm_b200_engine *e) { return e ? e->err : "null engine"; }

void *sddmm_b200_stream(sddmm_b200_engine *e) { return e ? static_cast<void *>(e->stream) : nullptr; }

int sddmm_b200_host_alloc(void **ptr, int64_t bytes) {
    if (!ptr || bytes < 0) return SDDMM_B200_ERR_ARG;
    cudaError_t st = cudaHostAlloc(ptr, static_cast<size_t>(std::max<int64_t>(bytes, 1)), cudaHostAllocDefault);
    if (st != cudaSuccess) {
        cudaGetLastError();
        *ptr = nullptr;
        return st == cudaErrorMemoryAllocation ? SDDMM_B200_ERR_OOM : SDDMM_B200_ERR_CUDA;
    }
    return SDDMM_B200_OK;
}

int sddmm_b200_host_free(void *ptr) {
    if (!ptr) return SDDMM_B200_OK;
    return cudaFreeHost(ptr) == cudaSuccess ? SDDMM_B200_OK : SDDMM_B200_ERR_CUDA;
}


// ---------------------------------------------------------------------------------------------
// Allocation-free SDDMM (see sddmm_b200_sddmm_csr_prealloc in the header).
//
// The row-tile kernel needs two pieces of scratch besides its operands: the table that says in which
// rows each nnz-balanced work item begins and ends, and an error word for its bounded waits.  Here
// both live in a fixed device array that is part of the loaded library image, so the call below never
// asks the CUDA allocator for anything.  The array name is only a host-side handle: its device address
// is looked up once per device with cudaGetSymbolAddress (that device current) and cached.
constexpr int64_t kPreallocMaxNnz = int64_t(1) << 27;                   // 134 217 728 nonzeros
constexpr int kPreallocItemNnz = 2048;
constexpr int64_t kPreallocMaxItems = kPreallocMaxNnz / kPreallocItemNnz;  // 65 536 work items
constexpr size_t kPreallocTableBytes = static_cast<size_t>(kPreallocMaxItems) * sizeof(int2);   // 512 KiB
constexpr size_t kPreallocScratchBytes = kPreallocTableBytes + 256;      // + the error word, on its own 256-byte line
static __device__ __align__(256) unsigned char g_prealloc_scratch[kPreallocScratchBytes];

constexpr int kPreallocMaxDevices = 64;
static unsigned char *g_prealloc_ptr[kPreallocMaxDevices] = {nullptr};   // device address of the array, per device

int sddmm_b200_sddmm_csr_prealloc(int device, void *cuda_stream, int64_t M, int64_t N, int64_t K, int64_t nnz,
                                  const int32_t *d_row_ptr, const int32_t *d_col_idx, const float *d_s_val,
                                  const float *d_A, const float *d_B, float *d_p_val) {
    if (M < 1 || N < 1 || K < 1 || nnz < 0 || device < 0 || device >= kPreallocMaxDevices) return SDDMM_B200_ERR_ARG;
    if (!d_row_ptr || !d_A || !d_B || (nnz > 0 && (!d_col_idx || !d_s_val || !d_p_val))) return SDDMM_B200_ERR_ARG;
    if (M >= (int64_t(1) << 31) - 1 || N >= (int64_t(1) << 31) - 1) return SDDMM_B200_ERR_ARG;
    // the kernel reads col_idx, A and B with 16-byte accesses (the engine's own arena is 256-byte aligned; a caller's
    // pointer into the middle of a larger buffer may not be) -- refused here rather than faulting on the GPU
    auto misaligned = [](const void *ptr, uintptr_t a) { return (reinterpret_cast<uintptr_t>(ptr) & (a - 1)) != 0; };
    if (misaligned(d_A, 16) || misaligned(d_B, 16) || (nnz > 0 && misaligned(d_col_idx, 16))) return SDDMM_B200_ERR_ARG;
    if (misaligned(d_row_ptr, 4) || (nnz > 0 && (misaligned(d_s_val, 4) || misaligned(d_p_val, 4)))) return SDDMM_B200_ERR_ARG;
    if (nnz > kPreallocMaxNnz) return SDDMM_B200_ERR_UNSUPPORTED;        // the work-item table would not fit the fixed scratch
    const int cpl = round_up_cpl(K);
    if (K % 4 != 0 || cpl == 0) return SDDMM_B200_ERR_UNSUPPORTED;      // only the row-tile kernel (K % 4 == 0, K <= 256) is offered here
    if (nnz == 0) return SDDMM_B200_OK;
    DeviceGuard g(device);
    if (!g.ok) return SDDMM_B200_ERR_CUDA;
    if (!g_prealloc_ptr[device]) {   // first call on this device: resolve the array's device address
        void *p = nullptr;
        if (cudaGetSymbolAddress(&p, g_prealloc_scratch) != cudaSuccess || !p) {
            cudaGetLastError();
            return SDDMM_B200_ERR_CUDA;
        }
        g_prealloc_ptr[device] = static_cast<unsigned char *>(p);
    }
    int2 *item_rows = reinterpret_cast<int2 *>(g_prealloc_ptr[device]);
    int32_t *err = reinterpret_cast<int32_t *>(g_prealloc_ptr[device] + kPreallocTableBytes);
    cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);

    const int n_items = static_cast<int>((nnz + kPreallocItemNnz - 1) / kPreallocItemNnz);
    // the array keeps whatever the previous call left: the error word must start at zero, the table is rewritten
    if (cudaMemsetAsync(err, 0, sizeof(int32_t), st) != cudaSuccess) return SDDMM_B200_ERR_CUDA;
    k_item_rows<<<grid_for(n_items, kBlock, 1 << 30), kBlock, 0, st>>>(d_row_ptr, static_cast<int32_t>(M), nnz, kPreallocItemNnz, n_items, item_rows);

    int64_t R = kPreallocItemNnz / std::max<int64_t>(1, nnz / M) + 1;
    R = (R + 7) / 8 * 8;
    R = std::max<int64_t>(1, std::min<int64_t>(std::min<int64_t>(R, kMaxStageBytes / (K * 4)), M));
    const int smem = static_cast<int>(rowtile_smem_bytes(static_cast<int>(R), static_cast<uint32_t>(K * 4)));
    const bool exact = (K == 32 * cpl);
    RowTileFn<float> fn = pick_rowtile<float>(cpl, exact);
    if (ensure_dynamic_smem_limit(reinterpret_cast<const void *>(fn), device, kRowTileMaxSmem)) return SDDMM_B200_ERR_CUDA;
    int occ = 0, sms = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, reinterpret_cast<const void *>(fn), kBlock, smem) != cudaSuccess || occ < 1) return SDDMM_B200_ERR_CUDA;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return SDDMM_B200_ERR_CUDA;

    RowTileArgs a;
    a.row_ptr = d_row_ptr; a.col_idx = d_col_idx; a.s_val = d_s_val; a.p_val = d_p_val; a.A = d_A; a.B = d_B;
    a.item_rows = item_rows; a.item_ids = nullptr; a.covered = nullptr;
    a.err = err; a.nnz = nnz; a.M = static_cast<int32_t>(M); a.K = static_cast<int32_t>(K);
    a.n_items = n_items; a.item_nnz = kPreallocItemNnz; a.rows_per_stage = static_cast<int32_t>(R);
    fn<<<std::min(n_items, sms * occ), kBlock, smem, st>>>(a);
    if (cudaGetLastError() != cudaSuccess) return SDDMM_B200_ERR_CUDA;
    int32_t h_err = 0;   // synchronous by contract: wait, then read the error word back
    if (cudaMemcpyAsync(&h_err, err, sizeof(int32_t), cudaMemcpyDeviceToHost, st) != cudaSuccess) return SDDMM_B200_ERR_CUDA;
    if (cudaStreamSynchronize(st) != cudaSuccess) return SDDMM_B200_ERR_CUDA;
    return h_err == kDevOk ? SDDMM_B200_OK : SDDMM_B200_ERR_DEVICE_WAIT;
}

}  // extern "C"

#include "pipeline.cuh"
