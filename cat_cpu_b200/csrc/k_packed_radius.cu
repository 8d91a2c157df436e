// k_packed_radius.cu -- K3: bit-packed LtL step (one bit per cell), the kernels of one
// radius (LTL_RADIUS; build.py compiles a part for each, see packed_ops.h).
//
// Same function as the reference's HostSolver<int> step (kezada94/CAT_cpu,
// src/CellularAutomata/Solvers/HostSolver.tpp:58-91, torus halo :93-140), with
// 32 cells per 32-bit word and the neighbour count kept bit-sliced:
//   h(row) = horizontal (2R+1)-window count of one row, as PH bit planes
//            (window_counts in packed_core.cuh);
//   B      = vertical sliding sum of h over 2R+1 rows, as PB bit planes
//            (B += h(r+R+1) - h(r-R) while a lane walks down its band);
//   next   = s ? [smin+1 <= B <= smax+1] : [bmin <= B <= bmax]   (B includes the centre)
// evaluated with bit-sliced comparators.  Every operation acts on 32 cells.
//
// Bound by the ALU pipe (16 lanes per scheduler and clock; measured 2.0 cycles per
// warp for lop3 and funnel shifts alike, and multiply-adds on the otherwise idle FMA
// pipe cannot do either).  At R = 5 a word costs 67 such operations: window count
// 23.5, moving B 21, rule 23.  Measured per generation at 16384^2, R = 5: 71.9 us
// before (a halo'd frame, one word per lane, neighbours by shuffle, 90 operations and
// as many again around them, 71% of the ALU), 43.5 now (81% in a cold launch).
#include <algorithm>

#include "grid_barrier.cuh"
#include "packed_core.cuh"
#include "packed_ops.h"
#include "packed_tile.cuh"

namespace ltl {

constexpr int kPackedWarps = 4;      // band walk: one warp per scheduler, so that k CTAs load all four alike
constexpr int kTileThreads = 512;
constexpr int kTileMaxRadius = 16;   // radii of the tile kernels
constexpr size_t kTileSmem = 220 * 1024;

// Words per lane of the band walk.  Two share their neighbours' loads and half the
// loop's bookkeeping (16384^2, us, one / two: R = 1 33 / 26, R = 5 58 / 43, R = 9 75.5 /
// 58.7, R = 12 84.3 / 72.8, R = 16 100.7 / 86.4).  Above R = 10 their ring leaves one CTA
// per SM, which only rows without ragged lanes stand (12001^2 R = 12 59 / 72, R = 10 54 /
// 49); above R = 16 it does not fit.
constexpr int packed_words(int R, bool ragged) { return R <= (ragged ? 10 : 16) ? 2 : 1; }
// Ring.  From R = 29 on it leaves one or two warps per SM, and counting the leaving row
// again is cheaper (16384^2 R = 32 216 us against 340 with one, R = 24 226 against 144).
template <int R>
constexpr bool packed_ring() { return R <= 28; }
// From R = 19 on the ring leaves one CTA per SM, whose four warps are too few to wait for
// memory: beyond the L2, and on rows with ragged lanes from half that size, large grids
// do without (us, ring / none: 32768^2 R = 20 868 / 617, R = 28 883 / 721; 33000^2 R = 20
// 1191 / 688; 20032^2 R = 28 303 / 281; 18496^2 R = 20 186 / 194, R = 28 201 / 235; 14001^2
// R = 19 153 / 129, R = 28 171 / 168; 12001^2 R = 19 113 / 99, R = 28 126 / 131).
constexpr bool packed_far_ringless(int R) { return R >= 19 && R <= 28; }

// Both frames of a grid against eighths of the L2.
static bool packed_beyond_l2(const PackedFrame& f, int eighths = 6) {  // (a rest of them stays in it)
    int dev = 0, l2 = 126 << 20;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&l2, cudaDevAttrL2CacheSize, dev);
    return 8ll * f.nrows() * f.wpitch > l2 / 8 * (long long)eighths;
}

// Rows in flight per lane: two where few warps share an SM (the larger rings) and the
// lane has no ragged words besides (16384^2 R = 8 58.9 -> 55.9, R = 12 72.7 -> 67.6, R = 5
// 43.4 -> 43.5; 12001^2 R = 16 68.5 -> 72.1).
constexpr bool packed_deep(int R, int W, int edge) { return edge == kEdgeNone && W == 2 && R >= 6; }

// Rows per band.  All bands of a step run at once, k CTAs on each SM, and each
// counts 2R+1 rows (at about 0.6 of an output row's cost) before its first output
// row: more CTAs per SM keep the ALU busier, fewer repeat less.  Time of a row
// relative to three or more CTAs per SM, measured on B200 at R = 5 (16384^2: 50.6,
// 44.6, 46.0 us at k = 2, 3, 4; 4096^2: k = 1 1.5 times): 1.5, 1.12, 1, 1.
//
// Small radii repeat little and wait for memory, so they take about 20 + 4R rows: as
// many CTAs as an SM holds, or several waves of them (one CTA more than it holds would
// be a wave of its own; 14001^2 R = 2 k = 5, 6, 7: 28.2, 30.8, 28.2 us).  us, long
// bands / these: 10001^2 R = 1 14.1 / 12.6; 16001^2 R = 1 33.2 / 26.7, R = 4 49.4 / 47.1
// (R = 5 no gain); 15040^2 R = 1 24.5 / 22.6; 16384^2 R = 3 35.8 / 36.5.  Beyond the L2
// long bands cost up to twice as much, every one of them being at another place of the
// grid: 32768^2 R = 1 173 / 91, R = 5 189 / 180; 20032^2 R = 1 61 / 40, R = 5 82 / 76;
// 22016^2 R = 6 93 / 97.
static int packed_band_rows(int rows, int groups, int R, bool ragged, bool beyond_l2, int sms, int per_sm) {
    static const double rate[] = {1.5, 1.12, 1.0, 1.0};
    double best = 0;
    int best_rows = rows;
    for (int k = 1; k <= std::min(per_sm, 4); ++k) {
        const long long bands = (long long)sms * k * kPackedWarps * 32 / groups;
        const int b = bands < 1 ? rows : std::max(2, (int)((rows + bands - 1) / bands));
        const double t = k * rate[k - 1] * (0.6 * (2 * R + 1) + b);
        if (best == 0 || t < best) {
            best = t;
            best_rows = b;
        }
    }
    const int brief = 20 + 4 * R;
    if (best_rows > brief && R <= (beyond_l2 ? 5 : ragged ? 4 : 2)) {
        const long long lanes = (long long)sms * kPackedWarps * 32;
        long long k = ((long long)rows * groups + brief * lanes - 1) / (brief * lanes);
        if (k == per_sm + 1) k = per_sm;
        const long long bands = std::max(1LL, k * lanes / groups);
        best_rows = std::min(best_rows, (int)((rows + bands - 1) / bands));
    }
    return std::min(best_rows, rows);
}

// Work split of a step: `groups` lanes along a row (W words each) by `bands` row
// bands, lanes numbered row by row.
struct PackedSplit {
    int groups, bands, band_rows;
    __device__ __forceinline__ bool item(int id, int rows, int W, int& w0, int& r0, int& r1) const {
        const int band = id / groups;
        if (band >= bands) return false;
        w0 = W * (id - band * groups);
        r0 = band * band_rows;
        r1 = min(r0 + band_rows, rows);
        return true;
    }
};

// One generation.  Two CTAs per SM are all that is asked of the compiler: left to
// itself it keeps to 64 registers and pays in instructions (16384^2 R = 8 77.5 us
// against 61.7, R = 12 91.9 / 84.7, R = 5 44.7 / 43.6).
template <int R, int W, bool kRing, int EDGE>
__global__ void __launch_bounds__(kPackedWarps * 32, 2)
k_packed_step(const uint32_t* __restrict__ cur, uint32_t* __restrict__ nxt, int wp, int n, int nw, int rows,
              PackedSplit split, const __grid_constant__ PackedRule pr) {
    extern __shared__ __align__(16) uint32_t ring_all[];
    uint32_t* ring = ring_all + (kRing ? (threadIdx.x >> 5) * PackedRing<R, W>::WARP_WORDS : 0);
    int w0, r0, r1;
    if (split.item(blockIdx.x * (kPackedWarps * 32) + threadIdx.x, rows, W, w0, r0, r1))
        packed_walk<R, W, kRing, EDGE, true, packed_deep(R, W, EDGE)>(cur, nxt, wp, n, nw, rows, r0, r1, w0, ring, threadIdx.x & 31, pr);
}

// `steps` generations in one cooperative launch, a tile per CTA (packed_tile.cuh), a
// grid barrier between generations.
struct TileSplit {
    int tile_rows, tile_words;  // of a tile (the last ones of the grid are smaller)
    int tiles_x, tiles;
};

template <int R, int EDGE>
__global__ void __launch_bounds__(kTileThreads, 1)
k_packed_tiles(uint32_t* a, uint32_t* b, int steps, int wp, int n, int nw, int rows, TileSplit split,
               const __grid_constant__ PackedRun run, const __grid_constant__ PackedRule pr) {
    extern __shared__ __align__(16) uint32_t counts[];
    GridBarrierWait all(run.barrier, gridDim.x, run.limit);
    const int step = kTileThreads / split.tile_words;  // rows of the tile that the CTA's threads take at once
    const int first = threadIdx.x / split.tile_words, col = threadIdx.x - first * split.tile_words;
    const int ty = blockIdx.x / split.tiles_x;
    const int r0 = ty * split.tile_rows, w0 = (blockIdx.x - ty * split.tiles_x) * split.tile_words + col;
    const int tr = min(split.tile_rows, rows - r0);
    const bool works = first < step && w0 < nw;
    const int band = (tr + step - 1) / step, b0 = first * band;
    for (int s = 0; s < steps; ++s) {
        const uint32_t* cur = s & 1 ? b : a;
        uint32_t* nxt = s & 1 ? a : b;
        if (works) tile_counts<R, EDGE, false>(cur, wp, n, nw, rows, r0, tr, w0, first, step, counts + col);
        __syncthreads();
        if (works && b0 < tr) tile_rows<R, false>(cur, nxt, wp, r0, b0, min(b0 + band, tr), w0, counts + col, pr);
        if (s + 1 < steps && !all.wait(run.err)) return;
    }
}

// The same for grids of at most kTileWords words per row: the generations are done
// in `blocks` blocks, and a CTA keeps its rows in shared memory for all d generations
// of a block.  It loads R d rows more on each side, and each generation is exact on R
// fewer of them.  A grid that is one CTA's alone (blocks = 1) wraps its rows in shared
// memory and needs no halo.  `blocks` is odd or even as `steps` is, so that the grid
// ends in the frame where single generations would have left it.
template <int R, int EDGE>
__global__ void __launch_bounds__(kTileThreads, 1)
k_packed_small(uint32_t* a, uint32_t* b, int steps, int blocks, int wp, int n, int nw, int rows, int band_rows,
               const __grid_constant__ PackedRun run, const __grid_constant__ PackedRule pr) {
    extern __shared__ __align__(16) uint32_t counts[];
    const bool whole = gridDim.x == 1;
    const int ext_max = whole ? rows : band_rows + 2 * R * block_generations(steps, blocks);
    uint32_t* s_in = counts + (size_t)(whole ? rows + 2 * R : ext_max) * PackedTile<R>::ROW;
    uint32_t* s_out = s_in + (size_t)ext_max * kTileStride;
    GridBarrierWait all(run.barrier, gridDim.x, run.limit);
    const int step = kTileThreads / nw;
    const int first = threadIdx.x / nw, col = threadIdx.x - first * nw;
    const bool works = first < step;
    const int r0 = blockIdx.x * band_rows, tr = min(band_rows, rows - r0);
    const uint32_t* cur = a;
    uint32_t* nxt = b;
    for (int s = 0; s < steps; --blocks) {
        const int d = block_generations(steps - s, blocks);
        const int halo = whole ? 0 : R * d, ext = tr + 2 * halo;
        if (works)
            for (int i = first; i < ext; i += step) {
                int r = r0 - halo + i;
                r += r < 0 ? rows : (r >= rows ? -rows : 0);
                s_in[i * kTileStride + col] = cur[(size_t)r * wp + col];
            }
        __syncthreads();
        for (int k = 1; k <= d; ++k) {
            const int lo = whole ? 0 : R * k, hi = whole ? rows : ext - R * k;
            if (works) tile_counts<R, EDGE, false>(s_in, kTileStride, n, nw, ext, lo, hi - lo, col, first, step, counts + col);
            __syncthreads();
            const int band = (hi - lo + step - 1) / step, b0 = first * band;
            if (works && b0 < hi - lo)
                tile_rows<R, false>(s_in, s_out, kTileStride, lo, b0, min(b0 + band, hi - lo), col, counts + col, pr);
            __syncthreads();
            uint32_t* t = s_in;
            s_in = s_out;
            s_out = t;
        }
        if (whole && steps % 2 == 0) nxt = a;  // (its only block, all read by now)
        if (works)
            for (int i = first; i < tr; i += step) nxt[(size_t)(r0 + i) * wp + col] = s_in[(halo + i) * kTileStride + col];
        s += d;
        if (s < steps && !all.wait(run.err)) return;
        const uint32_t* t = cur;
        cur = nxt;
        nxt = (uint32_t*)t;
    }
}

template <int R, int W, int EDGE, bool kRing = packed_ring<R>()>
struct PackedLaunch {
    static constexpr int smem = kRing ? kPackedWarps * PackedRing<R, W>::WARP_WORDS * 4 : 0;

    static cudaError_t prepare() {
        return cudaFuncSetAttribute(k_packed_step<R, W, kRing, EDGE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    smem);
    }
    template <class K>
    static PackedSplit split(K kernel, const PackedFrame& c, int band_rows, unsigned& ctas) {
        int dev = 0, sms = 148, per_sm = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kPackedWarps * 32, smem);
        const int rows = c.nrows(), groups = (c.nw + W - 1) / W;
        if (band_rows <= 0)
            band_rows = packed_band_rows(rows, groups, R, EDGE != kEdgeNone, packed_beyond_l2(c), sms, std::max(per_sm, 1));
        const int bands = (rows + band_rows - 1) / band_rows;
        const long long items = (long long)groups * bands;
        ctas = (unsigned)((items + kPackedWarps * 32 - 1) / (kPackedWarps * 32));
        return PackedSplit{groups, bands, band_rows};
    }
    static cudaError_t step(const PackedFrame& c, const PackedFrame& x, const PackedRule& pr, int band_rows,
                            cudaStream_t s) {
        auto kernel = k_packed_step<R, W, kRing, EDGE>;
        unsigned ctas;
        const PackedSplit sp = split(kernel, c, band_rows, ctas);
        kernel<<<ctas, kPackedWarps * 32, smem, s>>>(c.words, x.words, (int)c.wpitch, c.n, c.nw, c.nrows(), sp, pr);
        return cudaGetLastError();
    }
};

// A launch whose CTAs wait for one another (`waits`) has to be cooperative.
template <class... P, class... A>
static cudaError_t launch_group(void (*kernel)(P...), unsigned ctas, size_t smem, bool waits, cudaStream_t s,
                                A... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(ctas);
    cfg.blockDim = dim3(kTileThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeCooperative;
    at.val.cooperative = ctas > 1 && waits;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

template <int R, int EDGE>
struct TileLaunch {
    static cudaError_t prepare() {
        return cudaFuncSetAttribute(k_packed_tiles<R, EDGE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)kTileSmem);
    }
    // one tile per SM
    static TileSplit split(int rows, int nw, int sms) {
        TileSplit sp;
        const int tx = (nw + kTileWords - 1) / kTileWords;
        sp.tile_words = (nw + tx - 1) / tx;
        sp.tiles_x = (nw + sp.tile_words - 1) / sp.tile_words;
        const int bands = std::max(1, sms / sp.tiles_x);
        sp.tile_rows = (rows + bands - 1) / bands;
        sp.tiles = sp.tiles_x * ((rows + sp.tile_rows - 1) / sp.tile_rows);
        return sp;
    }
    static bool fits(int rows, int nw, int sms) {
        const TileSplit sp = split(rows, nw, sms);
        return sp.tiles <= sms && PackedTile<R>::bytes(sp.tile_rows) <= kTileSmem;
    }
    static cudaError_t run(const PackedFrame& c, const PackedFrame& x, const PackedRule& pr, int steps, int sms,
                           const PackedRun& run, cudaStream_t s) {
        const TileSplit sp = split(c.nrows(), c.nw, sms);
        return launch_group(k_packed_tiles<R, EDGE>, (unsigned)sp.tiles, PackedTile<R>::bytes(sp.tile_rows), steps > 1,
                            s, c.words, x.words, steps, (int)c.wpitch, c.n, c.nw, c.nrows(), sp, run, pr);
    }
};

template <int R, int EDGE>
struct SmallLaunch {
    static cudaError_t prepare() {
        return cudaFuncSetAttribute(k_packed_small<R, EDGE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)kTileSmem);
    }
    static size_t bytes(int rows, int tile_rows, int depth) {
        const int ext = tile_rows >= rows ? rows : tile_rows + 2 * R * depth;
        return PackedTile<R>::bytes(tile_rows >= rows ? rows : ext - 2 * R) + 2ull * ext * kTileStride * 4;
    }
    // rows per CTA: all SMs, but bands of at least 4 rows; grids of at most 256 words
    // are one CTA's (64^2 at R = 5: 0.78 us per generation against 1.03 in four bands
    // or more; 128^2 1.29 against 1.03)
    static int tile_rows(int rows, int nw, int sms) {
        return rows * nw <= 256 ? rows : std::min(rows, std::max(4, (rows + sms - 1) / sms));
    }
    static bool fits(int rows, int nw, int sms) {
        const int tr = tile_rows(rows, nw, sms);
        return nw <= kTileWords && bytes(rows, tr, 1) <= kTileSmem && (tr == rows || R <= rows);
    }
    static cudaError_t run(const PackedFrame& c, const PackedFrame& x, const PackedRule& pr, int steps, int sms,
                           const PackedRun& run, cudaStream_t s) {
        const int rows = c.nrows(), tr = tile_rows(rows, c.nw, sms);
        const unsigned ctas = (unsigned)((rows + tr - 1) / tr);
        // generations per block: a barrier and the reload cost about 1.5 us, a generation
        // 0.5 us and the rows that the tile has more.  Best measured (us per generation
        // at that depth and at 1): 1000^2 R = 2 1.33 at 6 (2.49), R = 5 2.19 at 4 (3.00),
        // R = 8 2.90 at 2 (3.38), R = 12 3.85 at 1; 128^2 R = 5 0.99 at 8 (2.31), R = 16
        // 2.48 at 2 (2.87)
        const int reach = c.nw <= 4 ? 28 : 18;
        int depth = std::min(steps, std::max(1, std::min(12, (2 * reach + R - 1) / (2 * R))));
        while (tr < rows && depth > 1 && (bytes(rows, tr, depth) > kTileSmem || R * depth > rows)) --depth;
        const int blocks = ctas == 1 ? 1 : run_blocks(steps, depth);
        depth = block_generations(steps, blocks);
        return launch_group(k_packed_small<R, EDGE>, ctas, bytes(rows, tr, depth), blocks > 1, s, c.words, x.words,
                            steps, blocks, (int)c.wpitch, c.n, c.nw, rows, tr, run, pr);
    }
};

// f(launcher) of the band walk's form for a grid.
template <int R, class F>
static cudaError_t with_walk(const PackedFrame& frame, F f) {
    const int n = frame.n;
    if constexpr (packed_far_ringless(R)) {
        const bool whole = packed_edge(n, 1) == kEdgeNone;
        if (n >= 64 && packed_beyond_l2(frame, whole ? 6 : 3))
            return whole ? f(PackedLaunch<R, 1, kEdgeNone, false>{}) : f(PackedLaunch<R, 1, kEdgeRagged, false>{});
    }
    if (!packed_two_words(n)) return f(PackedLaunch<R, 1, kEdgeTiny>{});
    if (packed_edge(n, 2) == kEdgeNone && packed_words(R, false) == 2)
        return f(PackedLaunch<R, packed_words(R, false), kEdgeNone>{});
    constexpr int W = packed_words(R, true);
    if (packed_edge(n, W) == kEdgeNone) return f(PackedLaunch<R, W, kEdgeNone>{});
    return f(PackedLaunch<R, W, kEdgeRagged>{});
}

template <int R>
cudaError_t PackedOps<R>::step(const PackedFrame& c, const PackedFrame& x, const PackedRule& pr, int band_rows,
                               cudaStream_t s) {
    return with_walk<R>(c, [&](auto l) { return l.step(c, x, pr, band_rows, s); });
}

// Which kernel advances a grid, by its words and R.  Measured per generation (us, 48
// per call; walk = one launch of the band walk each): 1024^2 R = 5 small 2.0, walk
// 4.4; 2048^2 R = 5 tiles 3.0, walk 5.4; 4096^2 R = 16 tiles 9.4, walk 15.3.  Tiles
// repeat 2R rows per tile and sum 2R+1 counts per thread, which the walk's long
// bands amortise on larger grids: at R = 1 and 2 the walk is ahead from 6400^2 on
// (6.9 against 7.4), at R = 3 to 12 tiles still are (9.2 / 10.3 to 15.5 / 22.1), and
// at 8192^2 the walk is (R = 5 15.3 against 27.6).
enum PackedRoute { kRouteWalk, kRouteTiles, kRouteSmall };

template <int R>
static PackedRoute packed_route_r(int rows, int nw, int sms) {
    if constexpr (R <= kTileMaxRadius) {
        if (SmallLaunch<R, kEdgeNone>::fits(rows, nw, sms)) return kRouteSmall;
        const long long words = (long long)rows * nw;
        if (words <= (R <= 2 ? 1000000 : 1280000) && TileLaunch<R, kEdgeNone>::fits(rows, nw, sms)) return kRouteTiles;
    }
    return kRouteWalk;
}

template <int R, int EDGE>
static cudaError_t prepare_packed_edge(PackedRoute route) {
    return route == kRouteSmall ? SmallLaunch<R, EDGE>::prepare() : TileLaunch<R, EDGE>::prepare();
}

template <int R, int EDGE>
static cudaError_t run_packed_edge(const PackedFrame& c, const PackedFrame& x, const PackedRule& pr, int steps,
                                   PackedRoute route, int sms, const PackedRun& run, cudaStream_t s) {
    return route == kRouteSmall ? SmallLaunch<R, EDGE>::run(c, x, pr, steps, sms, run, s)
                                : TileLaunch<R, EDGE>::run(c, x, pr, steps, sms, run, s);
}

template <int R>
cudaError_t PackedOps<R>::run(const PackedFrame& c, const PackedFrame& x, const PackedRule& pr, int steps, int sms,
                              const PackedRun& run, cudaStream_t s) {
    if constexpr (R <= kTileMaxRadius) {
        const PackedRoute route = packed_route_r<R>(c.nrows(), c.nw, sms);
        if (route == kRouteWalk) return cudaErrorInvalidValue;
        switch (packed_edge(c.n, 1)) {
            case kEdgeNone: return run_packed_edge<R, kEdgeNone>(c, x, pr, steps, route, sms, run, s);
            case kEdgeRagged: return run_packed_edge<R, kEdgeRagged>(c, x, pr, steps, route, sms, run, s);
            default: return run_packed_edge<R, kEdgeTiny>(c, x, pr, steps, route, sms, run, s);
        }
    }
    return cudaErrorInvalidValue;
}

// Attributes of the kernel that a grid's calls launch, and of no other: setting one loads
// the kernel.
template <int R>
bool PackedOps<R>::runs(const PackedFrame& f, int sms) {
    return packed_route_r<R>(f.nrows(), f.nw, sms) != kRouteWalk;
}

template <int R>
cudaError_t PackedOps<R>::prepare(const PackedFrame& f, bool walk, int sms) {
    if (walk) return with_walk<R>(f, [](auto l) { return l.prepare(); });
    if constexpr (R <= kTileMaxRadius) {
        const PackedRoute route = packed_route_r<R>(f.nrows(), f.nw, sms);
        if (route == kRouteWalk) return cudaErrorInvalidValue;
        switch (packed_edge(f.n, 1)) {
            case kEdgeNone: return prepare_packed_edge<R, kEdgeNone>(route);
            case kEdgeRagged: return prepare_packed_edge<R, kEdgeRagged>(route);
            default: return prepare_packed_edge<R, kEdgeTiny>(route);
        }
    }
    return cudaErrorInvalidValue;
}

#ifdef LTL_RADIUS
template struct PackedOps<LTL_RADIUS>;
#else
#define LTL_ALL(r) template struct PackedOps<r>;
LTL_PACKED_RADII(LTL_ALL)
#undef LTL_ALL
#endif

}  // namespace ltl
