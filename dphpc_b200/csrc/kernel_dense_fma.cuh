// Dense 64x64 tiles of S in plain fp32 arithmetic (fp32 mode): the tile's A and B rows are staged in shared memory once
// and every dot product of the tile is computed, in fp32 FMA, by a register-blocked loop; the nonzeros of S are then picked
// out by the tile's presence masks.  The gather kernels move one B row from L2 to the SM per nonzero -- 2 900 rows of 128
// bytes for a 70 %-full tile at K = 32 -- where this moves 128 rows and computes 30 % of the products for nothing:
// 18.07 M nonzeros in 64x64 blocks, K = 32 / 64 / 128: 73 / 112 / 194 us, against 143 / 259 / 468 us by gathers.
//
// A CTA of 128 threads is one tile at a time: thread (tx, ty) of 16 x 8 owns rows 8 ty .. 8 ty + 7 and columns tx, tx + 16,
// tx + 32, tx + 48.  For a fixed row the 16 lanes of a half-warp hold adjacent columns, so their S values are read and
// their P values written in pieces of one contiguous CSR run, straight from registers; S is requested before the last
// products are computed.  Operands arrive by cp.async one 32-column chunk of K ahead (the next tile's first chunk and its
// row descriptors while this tile's last chunk is computed).  Bound by FMA issue and the shared-memory reads beside it:
// 41 us per 32 columns where the FMA pipe alone needs 23.  Slower: 4 x 4 outputs on 256 threads (83 us at K = 32, twice the
// shared-memory reads), 8 x 8 on 64 threads (115, too few warps), packed fma.rn.f32x2 (79), 2 / 4 / 5 CTAs per SM (78 / 79 / 104).
#pragma once

#include "device_utils.cuh"
#include "kernel_dense_tile.cuh"

namespace sddmm {

struct DenseFmaArgs {
    const int2 *origins;          // n_tiles: {first row, first column}
    const DenseTileDesc *descs;   // n_tiles
    const float *s_val;
    float *p_val;
    const float *A;               // M x K
    const float *B;               // N x K
    int32_t n_tiles;
    int32_t M, N, K;              // K a multiple of 32
};

constexpr int kFmaThreads = 128;
constexpr int kFmaRowStride = 36;   // floats between staged rows: the 16-byte reads of either operand meet no bank twice

struct FmaSmem {
    float op[2][2][kDenseTile][kFmaRowStride];   // [buffer][A, B][row][k]
    DenseTileDesc desc[3];   // three: a warp may still read a tile's descriptor while another one requests that of the tile after next
};

template <bool OWN>
__global__ void __launch_bounds__(kFmaThreads, 3) sddmm_dense_tile_fma_kernel(const DenseFmaArgs args) {
    __shared__ __align__(16) FmaSmem sm;
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int chunks = args.K >> 5;

    // 32 columns of the 64 A rows and the 64 B rows of a tile (rows past the matrix repeat its last one: nothing samples them)
    auto stage_operands = [&](const int2 &o, int chunk, int buf) {
        const int part = tid & 7;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int side = q >> 2, row = (tid >> 3) + 16 * (q & 3);
            const int64_t r = side ? min(o.y + row, args.N - 1) : min(o.x + row, args.M - 1);
            cp_async_16(&sm.op[buf][side][row][4 * part], (side ? args.B : args.A) + r * args.K + 32 * chunk + 4 * part);
        }
    };
    auto stage_desc = [&](int tile, int buf) {
        static_assert(sizeof(DenseTileDesc) / 16 <= kFmaThreads, "one 16-byte copy per thread");
        if (tid < static_cast<int>(sizeof(DenseTileDesc) / 16))
            cp_async_16(reinterpret_cast<unsigned char *>(&sm.desc[buf]) + 16 * tid, reinterpret_cast<const unsigned char *>(args.descs + tile) + 16 * tid);
    };

    int tile = blockIdx.x;
    if (tile >= args.n_tiles) return;
    int2 origin = args.origins[tile];
    stage_desc(tile, 0);
    stage_operands(origin, 0, 0);
    cp_async_commit();
    int buf = 0, dbuf = 0;
    while (true) {
        const int next = tile + static_cast<int>(gridDim.x);
        const bool more = next < args.n_tiles;
        const int2 origin_next = more ? args.origins[next] : origin;
        // position in the CSR arrays of the nonzero (row 8 ty + i, column tx + 16 j), and whether this tile computes it
        auto locate = [&](int i, int j, int &pos) -> bool {
            const DenseTileDesc &d = sm.desc[dbuf];
            const int r = 8 * ty + i, c = (tx + 16 * j) & 31;
            const uint32_t lo = static_cast<uint32_t>(d.mask[r]), hi = static_cast<uint32_t>(d.mask[r] >> 32);
            const uint32_t word = j < 2 ? lo : hi;
            pos = d.start[r] + (j < 2 ? 0 : __popc(lo)) + __popc(word & ((1u << c) - 1u));
            const uint32_t mine = OWN ? static_cast<uint32_t>(d.own[r] >> (j < 2 ? 0 : 32)) : word;
            return (mine >> c) & 1u;
        };
        float acc[8][4], s[8][4];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                acc[i][j] = 0.f;
                s[i][j] = 0.f;
            }
        for (int chunk = 0; chunk < chunks; ++chunk) {
            // the next chunk (or the next tile's first) goes into the other buffer, whose readers are done (barrier below)
            if (chunk + 1 < chunks) {
                stage_operands(origin, chunk + 1, buf ^ 1);
            } else if (more) {
                stage_desc(next, dbuf == 2 ? 0 : dbuf + 1);
                stage_operands(origin_next, 0, buf ^ 1);
            }
            cp_async_commit();
            cp_async_wait_group<1>();
            __syncthreads();
            if (chunk == chunks - 1) {   // S, before the last products
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        int pos;
                        if (locate(i, j, pos)) s[i][j] = __ldcs(args.s_val + pos);
                    }
            }
            const float *a_base = &sm.op[buf][0][8 * ty][0], *b_base = &sm.op[buf][1][tx][0];
#pragma unroll 1
            for (int k = 0; k < 32; k += 4) {
                float4 a[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) a[i] = *reinterpret_cast<const float4 *>(a_base + i * kFmaRowStride + k);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float4 b = *reinterpret_cast<const float4 *>(b_base + 16 * j * kFmaRowStride + k);
#pragma unroll
                    for (int i = 0; i < 8; ++i) acc[i][j] = dot4(a[i], b, acc[i][j]);
                }
            }
            __syncthreads();
            buf ^= 1;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                int pos;
                if (locate(i, j, pos)) __stcs(args.p_val + pos, acc[i][j] * s[i][j]);
            }
        if (!more) break;
        tile = next;
        origin = origin_next;
        dbuf = dbuf == 2 ? 0 : dbuf + 1;
    }
    cp_async_wait_group<0>();
}

}  // namespace sddmm
