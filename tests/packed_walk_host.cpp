// The bit-packed band walk (cat_cpu_b200/csrc/packed_core.cuh) compiled for the
// host: one lane after the other, so that its arithmetic, its torus edges and
// every index it forms can be checked without a GPU (test_packed_walk.py).
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <vector>

#include <cuda_runtime.h>

static const uint32_t* g_lo;  // words a read may touch: [g_lo, g_hi)
static const uint32_t* g_hi;
static int g_bad;

template <class T>
static T __ldg(const T* p) {
    const uint32_t* q = (const uint32_t*)p;
    if (q < g_lo || q + sizeof(T) / 4 > g_hi || (uintptr_t)p % sizeof(T)) {
        ++g_bad;
        return T();
    }
    return *p;
}
static inline uint32_t __funnelshift_r(uint32_t lo, uint32_t hi, uint32_t s) {
    return (uint32_t)((((uint64_t)hi << 32) | lo) >> (s & 31));
}
static inline uint32_t __funnelshift_rc(uint32_t lo, uint32_t hi, uint32_t s) {
    return s >= 32 ? hi : (uint32_t)((((uint64_t)hi << 32) | lo) >> s);
}
static inline uint32_t __funnelshift_l(uint32_t lo, uint32_t hi, uint32_t s) {
    return (uint32_t)(((((uint64_t)hi << 32) | lo) << (s & 31)) >> 32);
}
static inline uint32_t __funnelshift_lc(uint32_t lo, uint32_t hi, uint32_t s) {
    return s >= 32 ? lo : (uint32_t)(((((uint64_t)hi << 32) | lo) << s) >> 32);
}

#include "packed_core.cuh"
#include "packed_tile.cuh"

using namespace ltl;

template <int R, int W, bool kRing, int EDGE>
static void grid_step(const uint32_t* cur, uint32_t* nxt, int wp, int n, int rows, int band_rows, const PackedRule& pr) {
    const int nw = (n + 31) / 32, groups = (nw + W - 1) / W;
    std::vector<uint4> ring((kRing ? PackedRing<R, W>::WARP_WORDS : 4) / 4 + 1);
    int lane = 0;
    for (int r0 = 0; r0 < rows; r0 += band_rows)
        for (int g = 0; g < groups; ++g, lane = (lane + 1) % 32)
            if (lane % 2)  // one or two rows in flight
                packed_walk<R, W, kRing, EDGE, true, true>(cur, nxt, wp, n, nw, rows, r0, std::min(r0 + band_rows, rows),
                                                           W * g, (uint32_t*)ring.data(), lane, pr);
            else
                packed_walk<R, W, kRing, EDGE, true>(cur, nxt, wp, n, nw, rows, r0, std::min(r0 + band_rows, rows), W * g,
                                                     (uint32_t*)ring.data(), lane, pr);
}

template <int R, bool kRing>
static int run(int words, const uint32_t* cur, uint32_t* nxt, int wp, int n, int rows, int band_rows,
               const PackedRule& pr) {
    if (words == 2 && !packed_two_words(n)) return 1;
    switch (packed_edge(n, words) + 3 * (words - 1)) {
        case 0: grid_step<R, 1, kRing, kEdgeNone>(cur, nxt, wp, n, rows, band_rows, pr); return 0;
        case 1: grid_step<R, 1, kRing, kEdgeRagged>(cur, nxt, wp, n, rows, band_rows, pr); return 0;
        case 2: grid_step<R, 1, kRing, kEdgeTiny>(cur, nxt, wp, n, rows, band_rows, pr); return 0;
        case 3: grid_step<R, 2, kRing, kEdgeNone>(cur, nxt, wp, n, rows, band_rows, pr); return 0;
        case 4: grid_step<R, 2, kRing, kEdgeRagged>(cur, nxt, wp, n, rows, band_rows, pr); return 0;
    }
    return 2;
}

// One generation of a rows x n torus of packed words (wp words per row), `words`
// words per lane.  Returns 0, 1 (form not used for this side), or 100 + the
// number of reads outside the grid.
extern "C" int packed_step_host(const uint32_t* cur, uint32_t* nxt, int wp, int n, int rows, int radius, int smin,
                                int smax, int bmin, int bmax, int words, int ring, int band_rows) {
    const PackedRule pr = make_packed_rule(Rule{radius, smin, smax, bmin, bmax});
    g_lo = cur;
    g_hi = cur + (size_t)rows * wp;
    g_bad = 0;
    int rc = 2;
    switch (radius) {
#define CASE(r)                                                                           \
    case r:                                                                               \
        rc = ring ? run<r, true>(words, cur, nxt, wp, n, rows, band_rows, pr)             \
                  : run<r, false>(words, cur, nxt, wp, n, rows, band_rows, pr);           \
        break;
        CASE(1) CASE(2) CASE(3) CASE(4) CASE(5) CASE(7) CASE(8) CASE(11) CASE(14) CASE(16) CASE(17) CASE(24) CASE(32)
    }
    return g_bad ? 100 + g_bad : rc;
}

// The tile form: tiles of tile_rows x tile_words, `threads` threads, output bands
// of band_rows rows.
template <int R, int EDGE>
static void tiles_step(const uint32_t* cur, uint32_t* nxt, int wp, int n, int rows, int tile_rows_, int tile_words,
                       int threads, int band_rows, const PackedRule& pr) {
    const int nw = (n + 31) / 32;
    for (int r0 = 0; r0 < rows; r0 += tile_rows_)
        for (int c0 = 0; c0 < nw; c0 += tile_words) {
            const int tr = std::min(tile_rows_, rows - r0), tc = std::min(tile_words, nw - c0);
            std::vector<uint32_t> h(PackedTile<R>::bytes(tr) / 4, 0xdeadbeefu);
            const int step = threads / tc;
            for (int t = 0; t < step * tc; ++t)
                tile_counts<R, EDGE, true>(cur, wp, n, nw, rows, r0, tr, c0 + t % tc, t / tc, step, h.data() + t % tc);
            for (int b0 = 0; b0 < tr; b0 += band_rows)
                for (int c = 0; c < tc; ++c)
                    tile_rows<R, true>(cur, nxt, wp, r0, b0, std::min(b0 + band_rows, tr), c0 + c, h.data() + c, pr);
        }
}

template <int R>
static int run_tiles(const uint32_t* cur, uint32_t* nxt, int wp, int n, int rows, int tr, int tc, int threads, int band,
                     const PackedRule& pr) {
    switch (packed_edge(n, 1)) {
        case kEdgeNone: tiles_step<R, kEdgeNone>(cur, nxt, wp, n, rows, tr, tc, threads, band, pr); break;
        case kEdgeRagged: tiles_step<R, kEdgeRagged>(cur, nxt, wp, n, rows, tr, tc, threads, band, pr); break;
        default: tiles_step<R, kEdgeTiny>(cur, nxt, wp, n, rows, tr, tc, threads, band, pr);
    }
    return 0;
}

extern "C" int packed_tiles_host(const uint32_t* cur, uint32_t* nxt, int wp, int n, int rows, int radius, int smin,
                                 int smax, int bmin, int bmax, int tr, int tc, int threads, int band) {
    const PackedRule pr = make_packed_rule(Rule{radius, smin, smax, bmin, bmax});
    g_lo = cur;
    g_hi = cur + (size_t)rows * wp;
    g_bad = 0;
    int rc = 2;
    switch (radius) {
#define TILE(r) \
    case r: rc = run_tiles<r>(cur, nxt, wp, n, rows, tr, tc, threads, band, pr); break;
        TILE(1) TILE(2) TILE(3) TILE(5) TILE(8) TILE(11) TILE(16)
    }
    return g_bad ? 100 + g_bad : rc;
}

// rule_planes against counts: the next state of a cell with box count `count`
// (centre included) and centre s, as the planes give it.
extern "C" int packed_rule_host(int radius, int smin, int smax, int bmin, int bmax, int count, int s) {
    const PackedRule pr = make_packed_rule(Rule{radius, smin, smax, bmin, bmax});
    const int M = 1 << planes_for_radius(radius);
    int init = 0;
    for (int i = 0; i < planes_for_radius(radius); ++i) init |= (pr.init[i] & 1) << i;
    const int v = (count + init) % M;
    uint32_t r = 0;
    switch (planes_for_radius(radius)) {
#define PLANES(p)                                                          \
    case p: {                                                              \
        uint32_t B[p];                                                     \
        for (int i = 0; i < p; ++i) B[i] = (v >> i & 1) ? ~0u : 0u;        \
        r = rule_planes<p>(B, s ? ~0u : 0u, pr);                           \
        break;                                                             \
    }
        PLANES(4) PLANES(5) PLANES(6) PLANES(7) PLANES(8) PLANES(9) PLANES(10) PLANES(11) PLANES(12) PLANES(13)
    }
    return r == 0u ? 0 : (r == ~0u ? 1 : -1);
}
