// Sizes the planner lays memory out by (dphpc_b200/csrc/plan_sizes.cuh): plain arithmetic, checked without a device.
#include <cstdint>

#include <algorithm>
#include <random>
#include <vector>

#include "check.hpp"
#include "plan_sizes.cuh"

TEST_CASE(tile_sums_hold_every_form_of_list_the_row_statistics_may_choose) {
    // around the lengths at which the tile grows, where a longer list has fewer tiles than a shorter one
    CHECK(sddmm::unit_tiles(600000) > sddmm::unit_tiles(1200000));
    for (int64_t edge : {int64_t(1) << 18, int64_t(1) << 20, int64_t(300000), int64_t(1) << 26})
        for (int64_t plain = 1; plain <= 8; ++plain)
            for (int64_t longs : {0, 2, 3, 8})
                for (int64_t part = 1; part <= 9; ++part)
                    for (int64_t off = -2; off <= 2; ++off) {
                        const int64_t M = edge / part + off, cap = sddmm::plan_tile_sums(M, plain, longs);
                        CHECK(cap >= sddmm::unit_tiles(M) && cap >= sddmm::unit_tiles(plain * M));
                        CHECK(cap >= sddmm::scan_tiles(M));
                        if (longs) CHECK(cap >= sddmm::unit_tiles((longs + 1) * M));
                    }
}

TEST_CASE(rows_without_copies_are_the_rows_of_the_matrix) {
    for (int64_t K = 1; K <= 400; ++K) {
        CHECK(sddmm::padded_row(false, K) >= K && sddmm::padded_row(false, K) % 8 == 0);
        CHECK(sddmm::padded_row(true, K) >= K && sddmm::padded_row(true, K) % 16 == 0);
        CHECK_EQ(sddmm::unpadded_row(K), K % 8 == 0 && K <= 256 ? K : 0);   // (K = 24, 40, 48, ... are padded otherwise)
    }
}

TEST_CASE(the_order_of_a_list_depends_on_that_list_alone) {
    // whole rows of an odd number of pieces are ordered, panels for their long rows are not; what the engine held before is no argument
    const double l2 = 126e6;
    for (int64_t row : {160, 224}) {
        CHECK(sddmm::by_size(false, row, false, 50e6, l2));
        CHECK(!sddmm::by_size(false, row, true, 50e6, l2));
    }
    for (int64_t row : {32, 64, 128, 256}) {
        CHECK(sddmm::by_size(false, row, false, sddmm::kPanelsFrom * l2, l2));
        CHECK(!sddmm::by_size(false, row, false, 0.86 * l2, l2));   // DRAM is the bound there
        CHECK(sddmm::by_size(false, row, true, 3 * l2, l2));
        CHECK(!sddmm::by_size(true, row, false, 50e6, l2));         // bf16
    }
    for (int64_t row : {8, 16, 24, 96}) CHECK(!sddmm::by_size(false, row, false, 50e6, l2));
}

TEST_CASE(building_a_list_loads_a_few_sums_per_tile_whatever_its_length) {
    for (int64_t rows : {int64_t(1) << 18, int64_t(2600000), int64_t(1) << 28})
        for (int64_t panels : {1, 3, 7}) {
            const int64_t tiles = sddmm::unit_tiles(rows * panels);
            const int64_t loads = tiles > sddmm::kDirectTiles ? 2 * tiles : tiles * tiles / 2;   // (scanned by one block first, or by each its own)
            CHECK(loads <= tiles * sddmm::kDirectTiles / 2);
            CHECK(tiles < (int64_t(1) << 31));
        }
}

TEST_CASE(residual_lists_cut_at_words_and_tiles_fit_the_capacity) {
    // 64 rows under `tiles` tiles: each tile owns 64 nonzeros of some rows and one of every other row, which cuts that row, so
    // that it owns just enough to stay; between two tiles a row holds `gap` nonzeros that are left over.  Lengths that start
    // rows and runs at every offset of a word, rows without tiles before and after.
    std::mt19937 rng(7);
    for (int tiles : {1, 2, 5, 40})
        for (int gap : {1, 2, 9, 33, 34, 66})
            for (int plain : {0, 1, 7, 32, 34, 64})
                for (int rep = 0; rep < 8; ++rep) {
                    std::vector<bool> covered;
                    int64_t rows = 0;
                    std::vector<int64_t> ends;   // of rows
                    auto add = [&](int n, bool c) { covered.insert(covered.end(), static_cast<size_t>(n), c); };
                    for (int r = 0; r < 100 + rep; ++r, ++rows) { add(plain ? std::max(1, plain + static_cast<int>(rng() % 3) - 1) : 0, false); ends.push_back(static_cast<int64_t>(covered.size())); }
                    std::vector<std::vector<int>> owned(static_cast<size_t>(tiles), std::vector<int>(64, 1));
                    for (auto &t : owned) {   // 16 rows of 61, 48 rows of 1: 1024
                        for (int r = 0; r < 16; ++r) t[static_cast<size_t>(r)] = 61;
                        std::shuffle(t.begin(), t.end(), rng);
                    }
                    for (int r = 0; r < 64; ++r, ++rows) {
                        for (int t = 0; t < tiles; ++t) { add(gap, false); add(owned[static_cast<size_t>(t)][static_cast<size_t>(r)], true); }
                        add(gap, false);
                        ends.push_back(static_cast<int64_t>(covered.size()));
                    }
                    int64_t units = 0, run = 0;
                    size_t e = 0;
                    const int64_t nnz = static_cast<int64_t>(covered.size());
                    for (int64_t j = 0; j <= nnz; ++j) {   // a run ends at a covered nonzero, the end of its row and the end of its word
                        bool cut = j == nnz || covered[static_cast<size_t>(j)] || j % 32 == 0;
                        while (e < ends.size() && ends[e] <= j) { cut = cut || ends[e] == j; ++e; }
                        if (cut) { units += (run + 7) / 8; run = 0; }
                        if (j < nnz && !covered[static_cast<size_t>(j)]) ++run;
                    }
                    CHECK(sddmm::kTileMinOwned == 16 * 61 + 48);
                    CHECK(units <= sddmm::unit_capacity(nnz, std::min(rows, nnz)));
                }
}

int main(int argc, char **argv) { return tiny_test::run_all(argc > 1 ? argv[1] : nullptr); }
