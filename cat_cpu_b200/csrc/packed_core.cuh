// packed_core.cuh -- bit-sliced building blocks shared by the packed kernels
// (single grid: k_packed_radius.cu, batched: k_batch.cu, k_batch_radius.cu).
//
// Cells are bits of 32-bit words (cell j of a row = bit j % 32 of word j / 32).
// A count over many cells is kept "bit-sliced": plane i holds bit i of the count
// of each of the 32 lanes, so one logic operation works on 32 cells.
#pragma once

#include <algorithm>
#include <type_traits>

#include "ltl_kernels.h"

// Radii of the bit-packed kernels (single grids; batches stop at 16).
#define LTL_BATCH_RADII(X) X(1) X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12) X(13) X(14) X(15) X(16)
#define LTL_PACKED_RADII(X)                                                                            \
    LTL_BATCH_RADII(X) X(17) X(18) X(19) X(20) X(21) X(22) X(23) X(24) X(25) X(26) X(27) X(28) X(29) X(30) \
    X(31) X(32)

namespace ltl {

__host__ __device__ constexpr int bits_for(int v) {
    int b = 0;
    while ((1 << b) <= v) ++b;
    return b;
}

// Three-input logic as single lop3 operations (the compiler does not always
// fuse these bit-sliced expressions into one instruction on its own):
//   xor3    a ^ b ^ c                       (sum of a full adder)     0x96
//   maj3    (a & b) | (a & c) | (b & c)     (carry of a full adder)   0xE8
//   borrow3 (~a & (b | c)) | (b & c)        (borrow out of a - b - c) 0x8E
// LTL_LOP3(table, the same function in C, for builds of this header without a GPU).
#ifdef __CUDACC__
#define LTL_LOP3(name, table, expr)                                                          \
    __device__ __forceinline__ uint32_t name(uint32_t a, uint32_t b, uint32_t c) {           \
        uint32_t d;                                                                          \
        asm("lop3.b32 %0, %1, %2, %3, " #table ";" : "=r"(d) : "r"(a), "r"(b), "r"(c));      \
        return d;                                                                            \
    }
#else
#define LTL_LOP3(name, table, expr) \
    inline uint32_t name(uint32_t a, uint32_t b, uint32_t c) { return expr; }
#endif
LTL_LOP3(xor3, 0x96, a ^ b ^ c)
LTL_LOP3(maj3, 0xE8, (a & b) | (a & c) | (b & c))
LTL_LOP3(borrow3, 0x8E, (~a & (b | c)) | (b & c))
// One step of each comparator chain as a single three-input logic operation
// (written as lop3 so that the run-time mask operand costs one instruction):
//   ge_step(m, b, ge) = m ? (b & ge) : (b | ge)
//   le_step(m, b, le) = m ? (~b | le) : (~b & le)
LTL_LOP3(ge_step, 0x8E, (a & (b & c)) | (~a & (b | c)))
LTL_LOP3(le_step, 0xB2, (a & (~b | c)) | (~a & (~b & c)))
#undef LTL_LOP3

// Wallace reduction: out[0..P) = bit planes of the number of set inputs per lane.
template <int M, int L, int P>
__device__ __forceinline__ void wallace(const uint32_t* v, uint32_t* out) {
    if constexpr (L < P) {
        if constexpr (M == 0) {
            out[L] = 0u;
            wallace<0, L + 1, P>(v, out);
        } else {
            constexpr int NF = (M >= 3) ? (M - 1) / 2 : 0;
            constexpr int REM = M - 2 * NF;
            constexpr int NH = (REM == 2) ? 1 : 0;
            constexpr int NC = NF + NH;
            uint32_t carry[NC > 0 ? NC : 1];
            uint32_t acc = v[0];
#pragma unroll
            for (int f = 0; f < NF; ++f) {
                uint32_t a = acc, b = v[1 + 2 * f], c = v[2 + 2 * f];
                acc = xor3(a, b, c);
                carry[f] = maj3(a, b, c);
            }
            if constexpr (NH == 1) {
                uint32_t b = v[M - 1];
                carry[NF] = acc & b;
                acc ^= b;
            }
            out[L] = acc;
            wallace<NC, L + 1, P>(carry, out);
        }
    }
}

// B += h
template <int PB, int PH>
__device__ __forceinline__ void planes_add(uint32_t (&B)[PB], const uint32_t (&h)[PH]) {
    uint32_t cy = 0u;
#pragma unroll
    for (int i = 0; i < PB; ++i) {
        const uint32_t b = B[i];
        if (i < PH) {
            B[i] = xor3(b, h[i], cy);
            cy = maj3(b, h[i], cy);
        } else {
            B[i] = b ^ cy;
            cy = b & cy;
        }
    }
}

constexpr int kMaxPlanes = 16;

// Interval rule on the box count B (centre included), for counts kept as
// B' = (B - o) mod 2^PB, o = the lower birth bound.  The offset costs nothing (B'
// starts at -o instead of 0) and turns the birth interval into one comparison,
// B' <= hi - lo; the survival interval needs two, [lo', hi'] modulo 2^PB, joined
// by AND, or by OR where the interval wraps.  Three carry chains instead of four,
// and no select for empty intervals: (2R+1)^2 <= 2^PB - 2 always (a square is not
// 2^k - 1 for k > 1), so an empty interval is the one value no count takes.
// Thresholds are per-plane masks (all-ones where the threshold's bit is set).
struct PackedRule {
    uint32_t init[kMaxPlanes];     // -o
    uint32_t birth_hi[kMaxPlanes];
    uint32_t live_lo[kMaxPlanes];
    uint32_t live_hi[kMaxPlanes];
    uint32_t live_wraps;           // ~0 where live_lo > live_hi
};

__host__ __device__ constexpr int planes_for_radius(int R) { return bits_for((2 * R + 1) * (2 * R + 1)); }

inline PackedRule make_packed_rule(const Rule& r) {
    const int maxB = (2 * r.radius + 1) * (2 * r.radius + 1);
    const int M = 1 << planes_for_radius(r.radius);
    const int blo = std::max(r.bmin, 0), bhi = std::min(r.bmax, maxB);
    // on B = k + 1 (clamped before the addition)
    const int slo = std::min(std::max(r.smin, -1), maxB) + 1, shi = std::min(r.smax, maxB - 1) + 1;
    const bool no_birth = blo > bhi, no_live = slo > shi;
    const int o = no_birth ? maxB + 1 : blo;
    const int width = no_birth ? 0 : bhi - blo;
    const int lo = ((no_live ? maxB + 1 : slo) - o + M) % M, hi = ((no_live ? maxB + 1 : shi) - o + M) % M;
    PackedRule p{};
    p.live_wraps = lo > hi ? 0xffffffffu : 0u;
    const int init = (M - o) % M;
    for (int i = 0; i < kMaxPlanes; ++i) {
        p.init[i] = ((init >> i) & 1) ? 0xffffffffu : 0u;
        p.birth_hi[i] = ((width >> i) & 1) ? 0xffffffffu : 0u;
        p.live_lo[i] = ((lo >> i) & 1) ? 0xffffffffu : 0u;
        p.live_hi[i] = ((hi >> i) & 1) ? 0xffffffffu : 0u;
    }
    return p;
}

// Next generation of 32 cells: B = planes of B', s = the centre cells.  Each
// chain is a carry out, from the least significant plane up: ge of B' + ~lo + 1,
// le of hi + ~B' + 1.
template <int PB>
__device__ __forceinline__ uint32_t rule_planes(const uint32_t (&B)[PB], uint32_t s, const PackedRule& pr) {
    uint32_t born = 0xffffffffu, ge = 0xffffffffu, le = 0xffffffffu;
#pragma unroll
    for (int i = 0; i < PB; ++i) {
        born = le_step(pr.birth_hi[i], B[i], born);
        ge = ge_step(pr.live_lo[i], B[i], ge);
        le = le_step(pr.live_hi[i], B[i], le);
    }
    const uint32_t lives = maj3(ge, le, pr.live_wraps);  // wraps ? ge | le : ge & le
    return (s & lives) | (~s & born);
}

// B += in - out for window counts in, out (mod 2^PB): one borrow chain over the
// PH planes, then one signed add.
template <int PB, int PH>
__device__ __forceinline__ void planes_move(uint32_t (&B)[PB], const uint32_t (&in)[PH], const uint32_t (&out)[PH]) {
    uint32_t d[PH], br = 0u;
#pragma unroll
    for (int i = 0; i < PH; ++i) {
        d[i] = xor3(in[i], out[i], br);
        br = borrow3(in[i], out[i], br);
    }
    uint32_t cy = 0u;
#pragma unroll
    for (int i = 0; i < PB; ++i) {
        const uint32_t b = B[i], x = i < PH ? d[i < PH ? i : 0] : br;  // br: the sign planes
        B[i] = xor3(b, x, cy);
        cy = maj3(b, x, cy);
    }
}

// ---------------------------------------------------------------------------
// Horizontal window counts h of W consecutive words of one row, given the word
// left of them, the words and the word right of them (x[0 .. W + 1]).
//
// R <= 3: a carry-save tree over the 2R+1 shifted copies of each word.
// R >= 4: the sums of three neighbouring cells are made once (one full adder on
// x shifted by 0, 1, 2: two planes) and shifted instead of the cells; windows of
// 2R+1 = 3 q + rest cells are the tree over q such sums and the rest.  The words
// are first moved by R cells, so that every shift goes one way and W + 1 words
// (W + 2 above R = 16) of sums serve W words of windows.  Operations per word at
// W = 2 (shifts and logic): R = 5 23.5 instead of 26, R = 8 37.5 instead of 46,
// R = 16 67 instead of 94.
// ---------------------------------------------------------------------------

// Carry-save tree whose weight-1 inputs are v0[M0] and weight-2 inputs v1[M1].
template <int M0, int M1, int P>
__device__ __forceinline__ void wallace2(const uint32_t (&v0)[M0], const uint32_t (&v1)[M1], uint32_t (&out)[P]) {
    constexpr int NF = (M0 - 1) / 2, NH = (M0 - 2 * NF == 2) ? 1 : 0, NC = NF + NH;
    uint32_t v[M1 + NC];
#pragma unroll
    for (int i = 0; i < M1; ++i) v[i] = v1[i];
    uint32_t acc = v0[0];
#pragma unroll
    for (int f = 0; f < NF; ++f) {
        v[M1 + f] = maj3(acc, v0[1 + 2 * f], v0[2 + 2 * f]);
        acc = xor3(acc, v0[1 + 2 * f], v0[2 + 2 * f]);
    }
    if constexpr (NH == 1) {
        v[M1 + NF] = acc & v0[M0 - 1];
        acc ^= v0[M0 - 1];
    }
    out[0] = acc;
    wallace<M1 + NC, 1, P>(v, out);
}

// Bits [32 w + o, 32 w + o + 32) of a row of words (o >= 0 at compile time).
template <int O, int N>
__device__ __forceinline__ uint32_t bits_from(const uint32_t (&v)[N], int w) {
    const int i = w + O / 32;
    if constexpr (O % 32 == 0) {
        return v[i];
    } else {
        return __funnelshift_r(v[i], i + 1 < N ? v[i + 1] : 0u, O % 32);
    }
}

template <int R, int W, int Q, int REST, int N>
struct WindowInputs {
    // weight-1 inputs: Q low planes at offsets 0, 3, .., REST raw cells after them
    template <int K>
    static __device__ __forceinline__ void low(const uint32_t (&y)[N], const uint32_t (&t0)[N], int w,
                                               uint32_t (&v)[Q + REST]) {
        if constexpr (K < Q) {
            v[K] = bits_from<3 * K>(t0, w);
            low<K + 1>(y, t0, w, v);
        } else if constexpr (K < Q + REST) {
            v[K] = bits_from<3 * Q + (K - Q)>(y, w);
            low<K + 1>(y, t0, w, v);
        }
    }
    template <int K>
    static __device__ __forceinline__ void high(const uint32_t (&t1)[N], int w, uint32_t (&v)[Q]) {
        if constexpr (K < Q) {
            v[K] = bits_from<3 * K>(t1, w);
            high<K + 1>(t1, w, v);
        }
    }
};

template <int R, int W, int PH>
__device__ __forceinline__ void window_counts(const uint32_t (&x)[W + 2], uint32_t (&h)[W][PH]) {
    if constexpr (R <= 3) {
#pragma unroll
        for (int w = 0; w < W; ++w) {
            uint32_t v[2 * R + 1];
#pragma unroll
            for (int d = -R; d <= R; ++d)
                v[d + R] = d == 0 ? x[w + 1]
                                  : (d > 0 ? __funnelshift_r(x[w + 1], x[w + 2], d) : __funnelshift_l(x[w], x[w + 1], -d));
            wallace<2 * R + 1, 0, PH>(v, h[w]);
        }
    } else {
        constexpr int N = W + (R <= 16 ? 1 : 2);
        constexpr int Q = (2 * R + 1) / 3, REST = (2 * R + 1) % 3;
        uint32_t y[N], t0[N], t1[N];  // y: cells from R before the word on; t0, t1: sums of three
#pragma unroll
        for (int i = 0; i < N; ++i) {
            if constexpr (R == 32) {
                y[i] = x[i];
            } else {
                y[i] = __funnelshift_r(x[i], i + 1 < W + 2 ? x[i + 1 < W + 2 ? i + 1 : 0] : 0u, 32 - R);
            }
        }
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const uint32_t nx = i + 1 < N ? y[i + 1 < N ? i + 1 : 0] : 0u;
            const uint32_t a = __funnelshift_r(y[i], nx, 1), b = __funnelshift_r(y[i], nx, 2);
            t0[i] = xor3(y[i], a, b);
            t1[i] = maj3(y[i], a, b);
        }
#pragma unroll
        for (int w = 0; w < W; ++w) {
            uint32_t v0[Q + REST], v1[Q];
            WindowInputs<R, W, Q, REST, N>::template low<0>(y, t0, w, v0);
            WindowInputs<R, W, Q, REST, N>::template high<0>(t1, w, v1);
            wallace2<Q + REST, Q, PH>(v0, v1, h[w]);
        }
    }
}

// ---------------------------------------------------------------------------
// The band walk: one lane advances W words of a row (from word w0 on) down the
// output rows [r0, r1).  B' (PB bit planes per word) slides down the band; the
// window counts h of the last 2R+1 rows wait in a ring in shared memory, private
// to the lane (kRing; else the leaving row is counted again).  Lanes do not talk
// to each other: the words left and right of the lane's come from memory (L1),
// so any mapping of lanes to (word group, band) works and no lane idles at the
// end of a row.  The torus is applied to the loads: rows wrap by index, and the
// first and last lane of a row take their neighbours from the row's other end
// (EDGE), so no frame has a halo and no pass refreshes one.  The next row's words
// are loaded one iteration ahead of their use.
//
// Joined rows.  Where 32 does not divide n (n >= 64), the last word's bits past n
// hold copies of the row's first cells.  An upload makes them so (join_word), and a
// step keeps them so at no cost: computed from joined words, the output bits past n
// are the next generation of those same first cells.  What is left of the edge is
// two funnel shifts per row, the same for every lane (by 32 and by 0 inside a row),
// so warps whose lanes are spread over rows do not diverge (a batch of 1024 grids of
// all sides: 82 ms per 256 generations with the edge lanes patched in branches, 62
// with joined rows).
// ---------------------------------------------------------------------------
enum PackedEdge {
    kEdgeNone = 0,    // 32 W divides n: neighbours are whole words
    kEdgeRagged = 1,  // a row's last lane holds cells past n (n >= 64, and nw > W); joined rows
    kEdgeTiny = 2     // n < 64 (W = 1): a row is at most two words, wrapped bit by bit
};

// Which form a side needs, for W words per lane.
__host__ __device__ inline int packed_edge(int n, int W) {
    return n < 64 ? kEdgeTiny : (n % (32 * W) == 0 ? kEdgeNone : kEdgeRagged);
}
// Two words per lane need a row of more than two words, or exactly two whole ones (one
// lane is the row's first and its last then).
__host__ __device__ inline bool packed_two_words(int n) { return n >= 64; }

// The ring of one warp: 2R+1 rows of PH planes of W words per lane, laid out so
// that a lane's planes are 16-byte vectors and a warp's vectors are contiguous.
template <int R, int W>
struct PackedRing {
    static constexpr int PH = bits_for(2 * R + 1);
    static constexpr int LANE_WORDS = PH * W;
    static constexpr int ROW_WORDS = LANE_WORDS * 32;
    static constexpr int WARP_WORDS = (2 * R + 1) * ROW_WORDS;

    static __device__ __forceinline__ void put(uint32_t* row, int lane, const uint32_t (&h)[W][PH]) {
        constexpr int V = LANE_WORDS / 4, REM = LANE_WORDS % 4;
#pragma unroll
        for (int v = 0; v < V; ++v)
            *(uint4*)(row + 128 * v + 4 * lane) =
                make_uint4(h[(4 * v) / PH][(4 * v) % PH], h[(4 * v + 1) / PH][(4 * v + 1) % PH],
                           h[(4 * v + 2) / PH][(4 * v + 2) % PH], h[(4 * v + 3) / PH][(4 * v + 3) % PH]);
        if constexpr (REM >= 2)
            *(uint2*)(row + 128 * V + 2 * lane) =
                make_uint2(h[(4 * V) / PH][(4 * V) % PH], h[(4 * V + 1) / PH][(4 * V + 1) % PH]);
        if constexpr (REM % 2 == 1)
            row[128 * V + (REM == 3 ? 64 : 0) + lane] = h[W - 1][PH - 1];
    }
    static __device__ __forceinline__ void get(const uint32_t* row, int lane, uint32_t (&h)[W][PH]) {
        constexpr int V = LANE_WORDS / 4, REM = LANE_WORDS % 4;
#pragma unroll
        for (int v = 0; v < V; ++v) {
            const uint4 q = *(const uint4*)(row + 128 * v + 4 * lane);
            h[(4 * v) / PH][(4 * v) % PH] = q.x;
            h[(4 * v + 1) / PH][(4 * v + 1) % PH] = q.y;
            h[(4 * v + 2) / PH][(4 * v + 2) % PH] = q.z;
            h[(4 * v + 3) / PH][(4 * v + 3) % PH] = q.w;
        }
        if constexpr (REM >= 2) {
            const uint2 q = *(const uint2*)(row + 128 * V + 2 * lane);
            h[(4 * V) / PH][(4 * V) % PH] = q.x;
            h[(4 * V + 1) / PH][(4 * V + 1) % PH] = q.y;
        }
        if constexpr (REM % 2 == 1) h[W - 1][PH - 1] = row[128 * V + (REM == 3 ? 64 : 0) + lane];
    }
};

// 32 cells from cell a on (0 <= a < n) of a periodic row of n < 64 cells whose
// first 64 bits are v (copies of the row from bit n on).
__device__ __forceinline__ uint32_t tiny_cells(uint64_t v, int n, int a) {
    // bits past 64 continue the period: cell 64 + i is cell 64 % n + i
    return (uint32_t)(a == 0 ? v : (v >> a) | ((v >> (64 % n)) << (64 - a)));
}

// The last word of a row of n cells (32 does not divide n, n >= 64), given its inner
// cells and the row's first word: joined.
__host__ __device__ inline uint32_t join_word(uint32_t last, uint32_t first, int n) {
    return (last & ((1u << (n & 31)) - 1u)) | (first << (n & 31));
}

// One row's words for a lane, as loaded: x[0] left, x[1 .. W] own, x[W + 1]
// right, e the extra word that an edge lane needs.  fix() turns them into the
// torus's words.
template <int W, int EDGE>
struct RowWords {
    uint32_t x[W + 2];
    uint32_t e = 0u;
};

template <int W, int EDGE, bool kConst>
struct RowReader {
    int n, nw, w0;
    int dl, dr, de;   // offsets of the left, right and extra word from the lane's first
    int sl, sr;       // shifts that join the extra word to the left and the right word
    bool edge;        // first or last lane of the row
    bool short_;      // W = 2: the row ends with the lane's first word

    __device__ __forceinline__ RowReader(int n_, int nw_, int w0_) : n(n_), nw(nw_), w0(w0_) {
        const int jl = nw - 1 - w0;          // index of the row's last word among the lane's own
        const int ib = n - 32 * (nw - 1);    // cells in the row's last word, 1..32
        dl = w0 == 0 ? nw - 1 : -1;
        dr = jl < W ? -w0 : W;
        de = w0 == 0 ? nw - 2 : 1 - w0;
        sl = w0 == 0 ? ib : 32;
        sr = jl < W ? 32 - ib : 0;
        edge = w0 == 0 || jl < W;
        short_ = W == 2 && jl == 0;
    }
    static __device__ __forceinline__ uint32_t ld(const uint32_t* p) {
        if constexpr (kConst) return __ldg(p);
        else return *p;
    }
    // p: the lane's first word in the row
    __device__ __forceinline__ void load(const uint32_t* p, RowWords<W, EDGE>& r) const {
        if constexpr (EDGE == kEdgeTiny) {
            r.x[1] = ld(p - w0);
            r.e = nw > 1 ? ld(p - w0 + 1) : 0u;
        } else {
            own(p, r.x + 1);
            r.x[0] = ld(p + dl);
            r.x[W + 1] = ld(p + dr);
            if constexpr (EDGE == kEdgeRagged)
                if (edge) r.e = ld(p + de);
        }
    }
    __device__ __forceinline__ void own(const uint32_t* p, uint32_t* o) const {
        if constexpr (W == 2) {
            uint2 q;
            if constexpr (kConst) q = __ldg((const uint2*)p);
            else q = *(const uint2*)p;
            o[0] = q.x;
            o[1] = q.y;
        } else {
#pragma unroll
            for (int j = 0; j < W; ++j) o[j] = ld(p + j);
        }
    }
    __device__ __forceinline__ void fix(RowWords<W, EDGE>& r) const {
        if constexpr (EDGE == kEdgeTiny) {
            uint64_t v = ((uint64_t)r.e << 32) | r.x[1];
            v &= (1ull << n) - 1ull;
            for (int p = n; p < 64; p *= 2) v |= v << p;
            const int a = (32 * w0) % n;
            r.x[0] = tiny_cells(v, n, (a + n - 32 % n) % n);
            r.x[1] = tiny_cells(v, n, a);
            r.x[2] = tiny_cells(v, n, (a + 32) % n);
        } else if constexpr (EDGE == kEdgeRagged) {
            // right: a last lane's is the row's start from cell 32 nw - n on; left: a
            // first lane's is cells n - 32 .. n - 1, the last word's inner cells and the
            // end of the word before.  (A first lane is never the last: nw > W.)
            const uint32_t right = __funnelshift_r(r.x[W + 1], r.e, sr);
            r.x[0] = __funnelshift_rc(r.e, r.x[0], sl);
            if constexpr (W == 2) r.x[2] = short_ ? right : r.x[2];
            r.x[W + 1] = right;
        }
    }
};

// cur, nxt: word 0 of row 0; wp words per row (a multiple of 4; the row's words
// up to a multiple of W may be written).  kConst: cur is not written while the
// kernel runs (read-only loads).  ring: this warp's ring.
template <int R, int W, bool kRing, int EDGE, bool kConst, bool kDeep = false>
__device__ __forceinline__ void packed_walk(const uint32_t* cur, uint32_t* nxt, int wp, int n, int nw, int rows, int r0,
                                            int r1, int w0, uint32_t* ring, int lane, const PackedRule& pr) {
    using Ring = PackedRing<R, W>;
    constexpr int PH = bits_for(2 * R + 1);
    constexpr int PB = planes_for_radius(R);
    const RowReader<W, EDGE, kConst> rd(n, nw, w0);
    const size_t all = (size_t)rows * wp;
    auto wrap = [&](const uint32_t*& p, int& r) {
        if (r == rows) {
            r = 0;
            p -= all;
        }
    };
    // entering row (ri, pi), leaving row (ro, po, without a ring), centre row, output row
    int ri = r0 - R < 0 ? r0 - R + rows : r0 - R, ro = ri;
    const uint32_t* pi = cur + (size_t)ri * wp + w0;
    const uint32_t* po = pi;
    const uint32_t* pc = cur + (size_t)r0 * wp + w0;
    uint32_t* pn = nxt + (size_t)r0 * wp + w0;
    uint32_t cen[W];
    rd.own(pc, cen);
    uint32_t B[W][PB];
#pragma unroll
    for (int w = 0; w < W; ++w)
#pragma unroll
        for (int i = 0; i < PB; ++i) B[w][i] = pr.init[i];
    uint32_t* slot = ring;
    // The window's first 2R+1 rows, kChunk loads in flight at a time: a band of a
    // few rows (a small grid) is little but this, and waits for L2 once per chunk.
    constexpr int kChunk = 4;
    auto start_rows = [&](auto count) {
        constexpr int kCount = decltype(count)::value;
        RowWords<W, EDGE> x[kCount];
#pragma unroll
        for (int k = 0; k < kCount; ++k) {
            rd.load(pi, x[k]);
            pi += wp;
            ++ri;
            wrap(pi, ri);
        }
#pragma unroll
        for (int k = 0; k < kCount; ++k) {
            rd.fix(x[k]);
            uint32_t h[W][PH];
            window_counts<R, W, PH>(x[k].x, h);
#pragma unroll
            for (int w = 0; w < W; ++w) planes_add<PB, PH>(B[w], h[w]);
            if constexpr (kRing) {
                Ring::put(slot, lane, h);
                slot += Ring::ROW_WORDS;
            }
        }
    };
#pragma unroll 1
    for (int k = 0; k < (2 * R + 1) / kChunk; ++k) start_rows(std::integral_constant<int, kChunk>{});
    if constexpr ((2 * R + 1) % kChunk != 0) start_rows(std::integral_constant<int, (2 * R + 1) % kChunk>{});
    slot = ring;
    const uint32_t* const ring_end = ring + Ring::WARP_WORDS;
    // rows in flight: the next one, kDeep also the one after it (and its centre)
    RowWords<W, EDGE> next, next2;
    uint32_t cen2[W];
    if (r0 + 1 < r1) rd.load(pi, next);
    if constexpr (kDeep) {
        pi += wp;
        ++ri;
        wrap(pi, ri);
        if (r0 + 2 < r1) rd.load(pi, next2);
        pc += wp;
        if (r0 + 1 < r1) rd.own(pc, cen2);
    }
#pragma unroll 1
    for (int r = r0;; ++r) {
        uint32_t val[W];
#pragma unroll
        for (int w = 0; w < W; ++w) val[w] = rule_planes<PB>(B[w], cen[w], pr);
        if constexpr (W == 2) {
            *(uint2*)pn = make_uint2(val[0], val[1]);
        } else {
#pragma unroll
            for (int w = 0; w < W; ++w) pn[w] = val[w];
        }
        if (r + 1 >= r1) break;
        pn += wp;
        pc += wp;
        RowWords<W, EDGE> x = next;
        pi += wp;
        ++ri;
        wrap(pi, ri);
        if constexpr (kDeep) {
#pragma unroll
            for (int w = 0; w < W; ++w) cen[w] = cen2[w];
            next = next2;
            if (r + 2 < r1) rd.own(pc, cen2);
            if (r + 3 < r1) rd.load(pi, next2);
        } else {
            rd.own(pc, cen);
            if (r + 2 < r1) rd.load(pi, next);
        }
        rd.fix(x);
        uint32_t in[W][PH], out[W][PH];
        if constexpr (kRing) {
            Ring::get(slot, lane, out);
        } else {
            RowWords<W, EDGE> y;
            rd.load(po, y);
            po += wp;
            ++ro;
            wrap(po, ro);
            rd.fix(y);
            window_counts<R, W, PH>(y.x, out);
        }
        window_counts<R, W, PH>(x.x, in);
#pragma unroll
        for (int w = 0; w < W; ++w) planes_move<PB, PH>(B[w], in[w], out[w]);
        if constexpr (kRing) {
            Ring::put(slot, lane, in);  // the entering row takes the leaving row's place
            slot += Ring::ROW_WORDS;
            if (slot == ring_end) slot = ring;
        }
    }
}

}  // namespace ltl
