// packed_tile.cuh -- the bit-packed generation of a tile by a whole CTA, for grids
// too small to fill the chip with long bands.
//
// The band walk (packed_core.cuh) counts 2R+1 rows before its first output row, one
// after the other: on a band of a few rows that is nearly all it does, and it is
// bound by the latency of that chain.  Here every row of the tile is counted once,
// by whichever thread, into shared memory (tile_counts); after a CTA barrier each
// thread sums the 2R+1 counts of its first output row in one carry-save tree, plane
// by plane, and slides from there (tile_rows).  A tile has at most 32 words per row
// (a warp on one row, or on several of a narrow grid).
#pragma once

#include "packed_core.cuh"

namespace ltl {

constexpr int kTileWords = 32;   // words per tile row at most
constexpr int kTileStride = 33;  // shared-memory words per plane of a row: rows of narrow tiles spread over the banks

// Blocks of generations between barriers: of `steps` generations, at most `depth` to a
// block.  Odd or even as `steps` is, so that the grid ends in the frame where single
// generations would have left it.
inline int run_blocks(int steps, int depth) {
    const int blocks = (steps + depth - 1) / depth;
    return blocks + (blocks % 2 != steps % 2);  // (more only where blocks < steps)
}
// Generations of the next block, with `left` of them in `blocks` blocks to come.
__host__ __device__ constexpr int block_generations(int left, int blocks) { return (left + blocks - 1) / blocks; }

template <int R>
struct PackedTile {
    static constexpr int PH = bits_for(2 * R + 1);
    static constexpr int PB = planes_for_radius(R);
    static constexpr int ROW = PH * kTileStride;  // words of one row's counts
    static constexpr size_t bytes(int tile_rows) { return (size_t)(tile_rows + 2 * R) * ROW * 4; }
};

// Counts of the tile's rows r0 - R .. r0 + tr - 1 + R at word w0, into h (the
// tile's counts at column `col`): this thread takes rows first, first + step, ..
template <int R, int EDGE, bool kConst>
__device__ __forceinline__ void tile_counts(const uint32_t* cur, int wp, int n, int nw, int rows, int r0, int tr,
                                            int w0, int first, int step, uint32_t* h) {
    using T = PackedTile<R>;
    constexpr int kLoads = 4;  // rows in flight per thread
    const RowReader<1, EDGE, kConst> rd(n, nw, w0);
    for (int i = first; i < tr + 2 * R; i += kLoads * step) {
        RowWords<1, EDGE> x[kLoads];
#pragma unroll
        for (int k = 0; k < kLoads; ++k) {
            const int j = i + k * step;
            int r = r0 - R + j;
            r += r < 0 ? rows : (r >= rows ? -rows : 0);
            if (j < tr + 2 * R) rd.load(cur + (size_t)r * wp + w0, x[k]);
        }
#pragma unroll
        for (int k = 0; k < kLoads; ++k) {
            const int j = i + k * step;
            if (j >= tr + 2 * R) break;
            rd.fix(x[k]);
            uint32_t c[1][T::PH];
            window_counts<R, 1, T::PH>(x[k].x, c);
#pragma unroll
            for (int p = 0; p < T::PH; ++p) h[(size_t)j * T::ROW + p * kTileStride] = c[0][p];
        }
    }
}

// Planes of init + the sum of 2R+1 consecutive rows' counts (mod 2^PB), from plane L
// up, with NC carries of weight L coming in.
template <int R, int L, int NC>
__device__ __forceinline__ void tile_sum(const uint32_t* h, const uint32_t* init, const uint32_t (&carry)[NC + 1],
                                         uint32_t (&B)[PackedTile<R>::PB]) {
    using T = PackedTile<R>;
    if constexpr (L < T::PB) {
        constexpr int ROWS = L < T::PH ? 2 * R + 1 : 0;
        constexpr int M = ROWS + NC + 1;
        constexpr int NF = (M - 1) / 2, NH = (M - 2 * NF == 2) ? 1 : 0;
        uint32_t v[M];
#pragma unroll
        for (int k = 0; k < ROWS; ++k) v[k] = h[k * T::ROW + L * kTileStride];
#pragma unroll
        for (int k = 0; k < NC; ++k) v[ROWS + k] = carry[k];
        v[M - 1] = init[L];
        uint32_t next[NF + NH + 1];
        uint32_t acc = v[0];
#pragma unroll
        for (int f = 0; f < NF; ++f) {
            next[f] = maj3(acc, v[1 + 2 * f], v[2 + 2 * f]);
            acc = xor3(acc, v[1 + 2 * f], v[2 + 2 * f]);
        }
        if constexpr (NH == 1) {
            next[NF] = acc & v[M - 1];
            acc ^= v[M - 1];
        }
        B[L] = acc;
        tile_sum<R, L + 1, NF + NH>(h, init, next, B);
    }
}

// Output rows [b0, b1) of the tile (tile-relative) at word w0; h as in tile_counts.
template <int R, bool kConst>
__device__ __forceinline__ void tile_rows(const uint32_t* cur, uint32_t* nxt, int wp, int r0, int b0, int b1, int w0,
                                          const uint32_t* h, const PackedRule& pr) {
    using T = PackedTile<R>;
    const uint32_t* pc = cur + (size_t)(r0 + b0) * wp + w0;
    uint32_t* pn = nxt + (size_t)(r0 + b0) * wp + w0;
    h += (size_t)b0 * T::ROW;
    uint32_t cen = RowReader<1, kEdgeNone, kConst>::ld(pc);
    uint32_t B[T::PB];
    const uint32_t none[1] = {0u};
    tile_sum<R, 0, 0>(h, pr.init, none, B);
#pragma unroll 1
    for (int j = b0;; ++j) {
        *pn = rule_planes<T::PB>(B, cen, pr);
        if (j + 1 >= b1) break;
        pn += wp;
        pc += wp;
        cen = RowReader<1, kEdgeNone, kConst>::ld(pc);
        uint32_t in[T::PH], out[T::PH];
#pragma unroll
        for (int p = 0; p < T::PH; ++p) {
            out[p] = h[p * kTileStride];
            in[p] = h[(2 * R + 1) * T::ROW + p * kTileStride];
        }
        planes_move<T::PB, T::PH>(B, in, out);
        h += T::ROW;
    }
}

}  // namespace ltl
