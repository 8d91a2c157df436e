// k_transfer.cu -- everything that moves a grid between its codings on the
// device: dense byte cells (a caller's buffer or a byte frame), the packed
// frame's 32-bit words, the PACK codec's 64-bit words; and the reductions over
// a grid (K6: population, comparison), read from whichever coding holds it.
//
// Every kernel here is bound by memory: a byte of cells in or out and an eighth
// of that in words.  So each thread moves whole 16-byte vectors of cells, in an
// order that keeps a warp's vectors contiguous, with kRows rows in flight per
// thread.  Callers' buffers may have any alignment and pitch: the kernels write
// vectors that are aligned in the destination, and read an unaligned source as
// aligned 32-bit words shifted together (load16).  Measured on B200, before
// (one byte, or 64 strided bytes, per thread) and after: 16384^2 cells to PACK
// words and back 2057 -> 107 us (604 MB, 5.6 TB/s; eight rows per thread 145);
// 16384^2 cells into a packed frame and out again 1376 -> 117 us (the byte frame
// between is gone too).
//
// Reference counterparts (kezada94/CAT_cpu): the host <-> solver copies of
// src/CellularAutomata/Solvers/AMXSolver.cpp (CASolver.cpp:3-13) and
// src/CellularAutomata/CADataDomainComparator.tpp:8-27.
#include <algorithm>

#include "grid_barrier.cuh"
#include "packed_core.cuh"
#include "transfer_core.cuh"

namespace ltl {

namespace {

constexpr int kTx = 32;    // threads along a row
constexpr int kTy = 8;     // rows per block pass
constexpr int kRows = 4;   // rows per thread in flight
// (Rows are counted unsigned: a grid of blocks may pass the last of 2^31 - 1 rows.)

// A block's threads along a row and rows: constants, unless rows are narrow (see shape;
// 16384^2 cells to words and back 113 us with them read from the launch, 107 so).
template <bool kNarrow>
__device__ __forceinline__ unsigned tx() { return kNarrow ? blockDim.x : kTx; }
template <bool kNarrow>
__device__ __forceinline__ unsigned ty() { return kNarrow ? blockDim.y : kTy; }

// A barrier that the grid's launches use, back to zero as the grid comes in.
__device__ __forceinline__ void reset_barrier(GridBarrier* barrier) {
    if (barrier && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0 && threadIdx.y == 0) barrier->arrived = 0;
}

// Rows on their way to the host after a wait may have run out (err: the word that this
// sets): the first cell, or 32 cells, become a mark, which tells the host to look.  The
// thread that stores them does it, last.
__device__ __forceinline__ bool marks(const unsigned int* err) {
    return err && blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0 && threadIdx.y == 0 && *err != 0u;
}

// 16-byte vectors that a row of cells may touch.
__host__ __device__ constexpr int vectors(int cols) { return (cols + 15) / 16 + 1; }

// Byte rows -> word rows: thread = one 32-bit word of a row, kNonzero: a cell is
// alive if its byte is not 0 (else by its bit 0).  Words past the cells get 0; bits
// past them in the last word 0, or the row's first cells (kJoin, cols >= 64).
template <bool kNonzero, bool kJoin, bool kNarrow>
__global__ void __launch_bounds__(kTx * kTy)
k_cells_to_words(const uint8_t* __restrict__ src, size_t sp, unsigned rows, int cols, uint32_t* __restrict__ dst, size_t dp,
                 int nwords, GridBarrier* barrier) {
    reset_barrier(barrier);
    const int w = blockIdx.x * tx<kNarrow>() + threadIdx.x;
    if (w >= nwords) return;
    const uint8_t* end = src + (size_t)(rows - 1) * sp + cols;
    const int valid = cols - 32 * w;
    const uint32_t mask = valid >= 32 ? 0xffffffffu : (valid > 0 ? (1u << valid) - 1u : 0u);
    for (unsigned r0 = blockIdx.y * (ty<kNarrow>() * kRows) + threadIdx.y; r0 < rows; r0 += gridDim.y * (ty<kNarrow>() * kRows)) {
        uint4 a[kRows], b[kRows];
#pragma unroll
        for (int k = 0; k < kRows; ++k) {
            const unsigned r = r0 + k * ty<kNarrow>();
            const uint8_t* p = src + (size_t)r * sp + 32 * (size_t)w;
            a[k] = b[k] = make_uint4(0u, 0u, 0u, 0u);
            if (r < rows && valid > 0) a[k] = load16<true>(p, src, end);
            if (r < rows && valid > 16) b[k] = load16<true>(p + 16, src, end);
        }
#pragma unroll
        for (int k = 0; k < kRows; ++k) {
            const unsigned r = r0 + k * ty<kNarrow>();
            if (r >= rows) continue;
            uint32_t v = (cells16_to_bits<kNonzero>(a[k]) | (cells16_to_bits<kNonzero>(b[k]) << 16)) & mask;
            if constexpr (kJoin) {
                if (valid > 0 && valid < 32) {
                    const uint8_t* p = src + (size_t)r * sp;
                    v = join_word(v, cells16_to_bits<kNonzero>(load16<true>(p, src, end)) |
                                         (cells16_to_bits<kNonzero>(load16<true>(p + 16, src, end)) << 16), cols);
                }
            }
            dst[(size_t)r * dp + w] = v;
        }
    }
}

// Word rows -> byte rows: thread = one aligned 16-byte vector of the destination.  (The mark
// is a form of its own: with its test in all, 4000^2 words to cells took 7.2 us, not 6.2.)
template <bool kNarrow, bool kMarked>
__global__ void __launch_bounds__(kTx * kTy)
k_words_to_cells(const uint32_t* __restrict__ src, size_t sp, int nwords, unsigned rows, int cols, uint8_t* __restrict__ dst,
                 size_t dp, const unsigned int* err) {
    const int v = blockIdx.x * tx<kNarrow>() + threadIdx.x;
    if (v >= vectors(cols)) return;
    for (unsigned r0 = blockIdx.y * (ty<kNarrow>() * kRows) + threadIdx.y; r0 < rows; r0 += gridDim.y * (ty<kNarrow>() * kRows)) {
        uint32_t bits[kRows];
#pragma unroll
        for (int k = 0; k < kRows; ++k) {
            const unsigned r = r0 + k * ty<kNarrow>();
            const int c = lead(dst + (size_t)r * dp) + 16 * v;
            bits[k] = r < rows && c < cols ? bits16_at(src + (size_t)r * sp, c, nwords) : 0u;
        }
#pragma unroll
        for (int k = 0; k < kRows; ++k) {
            const unsigned r = r0 + k * ty<kNarrow>();
            if (r >= rows) continue;
            uint8_t* row = dst + (size_t)r * dp;
            const int c = lead(row) + 16 * v;
            if (c < cols) store16<true>(row + c, bits16_to_cells(bits[k]), -c, cols - c);
        }
    }
    if (kMarked && marks(err)) dst[0] = kMarkCell;
}

// Byte rows -> byte rows (kNonzero: every byte that is not 0 becomes 1).
// src == dst is allowed: a thread reads only the vectors it writes.
template <bool kNonzero, bool kNarrow>
__global__ void __launch_bounds__(kTx * kTy)
k_copy_cells(const uint8_t* src, size_t sp, unsigned rows, int cols, uint8_t* dst, size_t dp) {
    const int v = blockIdx.x * tx<kNarrow>() + threadIdx.x;
    if (v >= vectors(cols)) return;
    const uint8_t* end = src + (size_t)(rows - 1) * sp + cols;
    for (unsigned r0 = blockIdx.y * (ty<kNarrow>() * kRows) + threadIdx.y; r0 < rows; r0 += gridDim.y * (ty<kNarrow>() * kRows)) {
        uint4 a[kRows];
#pragma unroll
        for (int k = 0; k < kRows; ++k) {
            const unsigned r = r0 + k * ty<kNarrow>();
            const int c = lead(dst + (size_t)r * dp) + 16 * v;
            a[k] = make_uint4(0u, 0u, 0u, 0u);
            if (r < rows && c < cols) a[k] = load16<false>(src + (size_t)r * sp + c, src, end);
        }
#pragma unroll
        for (int k = 0; k < kRows; ++k) {
            const unsigned r = r0 + k * ty<kNarrow>();
            if (r >= rows) continue;
            uint8_t* row = dst + (size_t)r * dp;
            const int c = lead(row) + 16 * v;
            if constexpr (kNonzero)
                a[k] = make_uint4(nonzero4(a[k].x), nonzero4(a[k].y), nonzero4(a[k].z), nonzero4(a[k].w));
            if (c < cols) store16<false>(row + c, a[k], -c, cols - c);
        }
    }
}

// Rows of a grid as 16-cell groups, from the byte frame (kWords = false) or the
// packed frame.  Cells past n read as 0.
struct GridRows {
    const void* inner;  // cell (0, 0): byte frame (16-byte aligned rows) or word frame
    size_t pitch;       // bytes or words
    int n;
    unsigned rows;
};

__device__ __forceinline__ void keep_cells(uint4& v, int valid) {
    if (valid >= 16) return;
    uint32_t q[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const int left = valid - 4 * k;
        q[k] = left >= 4 ? q[k] : (left > 0 ? q[k] & ((1u << (8 * left)) - 1u) : 0u);
    }
    v = make_uint4(q[0], q[1], q[2], q[3]);
}

template <bool kWords>
__global__ void __launch_bounds__(kTx * kTy) k_population(GridRows g, unsigned long long* out) {
    unsigned long long acc = 0;
    constexpr int kCells = kWords ? 32 : 16;
    const int v = blockIdx.x * kTx + threadIdx.x;
    const int valid = g.n - kCells * v;
    if (valid > 0) {
        for (unsigned r0 = blockIdx.y * (kTy * kRows) + threadIdx.y; r0 < g.rows; r0 += gridDim.y * (kTy * kRows)) {
            uint32_t cnt = 0;
#pragma unroll
            for (int k = 0; k < kRows; ++k) {
                const unsigned r = r0 + k * kTy;
                if (r >= g.rows) continue;
                if constexpr (kWords) {
                    uint32_t w = __ldg((const uint32_t*)g.inner + (size_t)r * g.pitch + v);
                    if (valid < 32) w &= (1u << valid) - 1u;
                    cnt += __popc(w);
                } else {
                    // the vector may reach into the right halo: those cells are dropped
                    uint4 a = __ldg((const uint4*)((const uint8_t*)g.inner + (size_t)r * g.pitch) + v);
                    keep_cells(a, valid);
                    cnt += __popc(a.x) + __popc(a.y) + __popc(a.z) + __popc(a.w);  // 0/1 bytes
                }
            }
            acc += cnt;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
    if (threadIdx.x == 0 && acc) atomicAdd(out, acc);
}

template <bool kWords>
__global__ void __launch_bounds__(kTx * kTy)
k_compare(GridRows g, const uint8_t* __restrict__ other, size_t op, unsigned long long* out) {
    unsigned long long cnt = 0, first = ~0ull;
    const int v = blockIdx.x * kTx + threadIdx.x;
    const int valid = g.n - 16 * v;
    if (valid > 0) {
        const uint8_t* end = other + (size_t)(g.rows - 1) * op + g.n;
        for (unsigned r0 = blockIdx.y * (kTy * kRows) + threadIdx.y; r0 < g.rows; r0 += gridDim.y * (kTy * kRows)) {
            uint4 a[kRows], b[kRows];
#pragma unroll
            for (int k = 0; k < kRows; ++k) {
                const unsigned r = r0 + k * kTy;
                a[k] = b[k] = make_uint4(0u, 0u, 0u, 0u);
                if (r >= g.rows) continue;
                if constexpr (kWords) {
                    const uint32_t w = __ldg((const uint32_t*)g.inner + (size_t)r * g.pitch + (v >> 1));
                    a[k] = bits16_to_cells((v & 1) ? w >> 16 : w & 0xffffu);
                } else {
                    a[k] = __ldg((const uint4*)((const uint8_t*)g.inner + (size_t)r * g.pitch) + v);
                }
                b[k] = load16<true>(other + (size_t)r * op + 16 * (size_t)v, other, end);
            }
#pragma unroll
            for (int k = 0; k < kRows; ++k) {
                uint4 d = make_uint4(nonzero4(a[k].x ^ b[k].x), nonzero4(a[k].y ^ b[k].y), nonzero4(a[k].z ^ b[k].z),
                                     nonzero4(a[k].w ^ b[k].w));
                keep_cells(d, valid);
                const uint32_t bits = cells16_to_bits<false>(d);
                if (bits) {
                    cnt += __popc(bits);
                    const unsigned long long at =
                        (unsigned long long)(r0 + k * kTy) * g.n + 16 * (unsigned)v + __ffs(bits) - 1;
                    first = at < first ? at : first;
                }
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        cnt += __shfl_down_sync(0xffffffffu, cnt, o);
        const unsigned long long f2 = __shfl_down_sync(0xffffffffu, first, o);
        first = f2 < first ? f2 : first;
    }
    if (threadIdx.x == 0 && cnt) {
        atomicAdd(out, cnt);
        atomicMin(out + 1, first);
    }
}

// Inner words of a packed frame -> PACK-coded rows (uint64 word k of a row =
// frame words 2k and 2k + 1), bits past n cleared.  Thread = one frame word.
template <bool kNarrow>
__global__ void __launch_bounds__(kTx * kTy)
k_words_to_pack(const uint32_t* __restrict__ src, size_t sp, unsigned rows, int n, uint32_t* __restrict__ dst, size_t dp,
                int nwords, const unsigned int* err) {
    const int w = blockIdx.x * tx<kNarrow>() + threadIdx.x;
    if (w >= nwords) return;
    const int valid = n - 32 * w;
    const uint32_t mask = valid >= 32 ? 0xffffffffu : (valid > 0 ? (1u << valid) - 1u : 0u);
    for (unsigned r = blockIdx.y * ty<kNarrow>() + threadIdx.y; r < rows; r += gridDim.y * ty<kNarrow>())
        dst[(size_t)r * dp + w] = valid > 0 ? __ldg(src + (size_t)r * sp + w) & mask : 0u;
    if (marks(err)) dst[0] = kMarkCells;
}

// The other way, last words joined (kJoin).
template <bool kJoin, bool kNarrow>
__global__ void __launch_bounds__(kTx * kTy)
k_pack_to_words(const uint32_t* __restrict__ src, size_t sp, unsigned rows, int n, uint32_t* __restrict__ dst, size_t dp,
                int nwords, GridBarrier* barrier) {
    reset_barrier(barrier);
    const int w = blockIdx.x * tx<kNarrow>() + threadIdx.x;
    if (w >= nwords) return;
    for (unsigned r = blockIdx.y * ty<kNarrow>() + threadIdx.y; r < rows; r += gridDim.y * ty<kNarrow>()) {
        uint32_t v = __ldg(src + (size_t)r * sp + w);
        if (kJoin && w == nwords - 1) v = join_word(v, __ldg(src + (size_t)r * sp), n);
        dst[(size_t)r * dp + w] = v;
    }
}

// Grid and block of a kernel without a reduction: `items` threads along a row, `per` rows per
// thread.  Where rows of a few cells would leave a warp to one or two threads, and are more
// than the SMs take at once, a block has fewer threads along a row (a power of two; 100,000
// rows of 3 cells packed 26 us with a warp per row, 10 so; a pass over 64^2 15.0 / 15.7).
struct Shape {
    dim3 grid, block;
    bool narrow;
};
Shape shape(long long items, int rows, int per) {
    unsigned tx = kTx;
    if (rows > 148 * 8 * kTy * per)
        while (tx > 1 && tx / 2 >= items) tx /= 2;
    const unsigned ty = kTx * kTy / tx;
    const long long gy = std::max<long long>(1, ((long long)rows + ty * per - 1) / (ty * per));
    return {dim3((unsigned)std::max<long long>(1, (items + tx - 1) / tx), (unsigned)std::min<long long>(gy, 65535)),
            dim3(tx, ty), tx < kTx};
}

// The same for a reduction, whose warps are rows; `cap` bounds its blocks (each ends in an
// atomic).
dim3 cover(long long items, int rows, int per, long long cap) {
    const long long gx = std::max<long long>(1, (items + kTx - 1) / kTx);
    long long gy = std::max<long long>(1, ((long long)rows + kTy * per - 1) / (kTy * per));
    gy = std::min(gy, std::max<long long>(1, cap / gx));
    return dim3((unsigned)gx, (unsigned)std::min<long long>(gy, 65535));
}

auto cells_to_words(bool nonzero, bool join, bool narrow) {
    if (narrow)
        return nonzero ? (join ? k_cells_to_words<true, true, true> : k_cells_to_words<true, false, true>)
                       : (join ? k_cells_to_words<false, true, true> : k_cells_to_words<false, false, true>);
    return nonzero ? (join ? k_cells_to_words<true, true, false> : k_cells_to_words<true, false, false>)
                   : (join ? k_cells_to_words<false, true, false> : k_cells_to_words<false, false, false>);
}

const dim3 kBlock(kTx, kTy);
constexpr long long kReduceBlocks = 148 * 16;

GridRows byte_rows(const Frame& f) {
    return GridRows{f.base + (size_t)f.H * f.pitch + f.H, f.pitch, f.n, (unsigned)f.nrows()};
}
uint32_t* word_origin(const PackedFrame& f) { return f.words + (size_t)f.HR * f.wpitch + f.HW; }
GridRows word_rows(const PackedFrame& f) { return GridRows{word_origin(f), f.wpitch, f.n, (unsigned)f.nrows()}; }

}  // namespace

// --- byte buffers <-> byte frames -------------------------------------------
cudaError_t launch_copy_in(const Frame& f, const uint8_t* src, size_t src_pitch, cudaStream_t s) {
    const int rows = f.nrows();
    const Shape b = shape(vectors(f.n), rows, kRows);
    (b.narrow ? k_copy_cells<true, true> : k_copy_cells<true, false>)<<<b.grid, b.block, 0, s>>>(src, src_pitch, rows, f.n,
                                                                                 f.inner(0, 0), f.pitch);
    return cudaGetLastError();
}

cudaError_t launch_copy_out(const Frame& f, uint8_t* dst, size_t dst_pitch, cudaStream_t s) {
    const int rows = f.nrows();
    const Shape b = shape(vectors(f.n), rows, kRows);
    (b.narrow ? k_copy_cells<false, true> : k_copy_cells<false, false>)<<<b.grid, b.block, 0, s>>>(f.cinner(0, 0), f.pitch, rows, f.n,
                                                                                  dst, dst_pitch);
    return cudaGetLastError();
}

// --- byte buffers <-> packed frames -----------------------------------------
cudaError_t launch_pack_rows(const uint8_t* src, size_t pitch, bool nonzero, const PackedFrame& dst, int row0,
                             int nrows, GridBarrier* barrier, cudaStream_t s) {
    if (nrows <= 0) return cudaSuccess;
    uint32_t* d = word_origin(dst) + (size_t)row0 * dst.wpitch;
    const bool join = dst.n >= 64 && dst.n % 32 != 0;
    const Shape b = shape(dst.nw, nrows, kRows);
    auto kernel = cells_to_words(nonzero, join, b.narrow);
    kernel<<<b.grid, b.block, 0, s>>>(src, pitch, nrows, dst.n, d, dst.wpitch, dst.nw,
                                                              barrier);
    return cudaGetLastError();
}

cudaError_t launch_unpack_rows(const PackedFrame& src, int row0, int nrows, uint8_t* dst, size_t pitch,
                               const unsigned int* err, cudaStream_t s) {
    if (nrows <= 0) return cudaSuccess;
    const Shape b = shape(vectors(src.n), nrows, kRows);
    auto kernel = err ? (b.narrow ? k_words_to_cells<true, true> : k_words_to_cells<false, true>)
                      : (b.narrow ? k_words_to_cells<true, false> : k_words_to_cells<false, false>);
    kernel<<<b.grid, b.block, 0, s>>>(
        word_origin(src) + (size_t)row0 * src.wpitch, src.wpitch, src.nw, nrows, src.n, dst, pitch, err);
    return cudaGetLastError();
}

// --- PACK codec ---------------------------------------------------------------
cudaError_t launch_pack(const uint8_t* cells, size_t cell_pitch, int rows, int cols, uint64_t* words,
                        size_t word_pitch_words, cudaStream_t s) {
    if (rows == 0 || cols == 0) return cudaSuccess;
    const int nwords = 2 * ((cols + 63) / 64);  // 32-bit halves, little-endian
    const Shape b = shape(nwords, rows, kRows);
    (b.narrow ? k_cells_to_words<true, false, true> : k_cells_to_words<true, false, false>)<<<b.grid, b.block, 0, s>>>(cells, cell_pitch, rows, cols,
                                                                       (uint32_t*)words, 2 * word_pitch_words, nwords,
                                                                       nullptr);
    return cudaGetLastError();
}

cudaError_t launch_unpack(const uint64_t* words, size_t word_pitch_words, int rows, int cols, uint8_t* cells,
                          size_t cell_pitch, cudaStream_t s) {
    if (rows == 0 || cols == 0) return cudaSuccess;
    const Shape b = shape(vectors(cols), rows, kRows);
    (b.narrow ? k_words_to_cells<true, false> : k_words_to_cells<false, false>)<<<b.grid, b.block, 0, s>>>(
        (const uint32_t*)words, 2 * word_pitch_words, 2 * ((cols + 63) / 64), rows, cols, cells, cell_pitch,
        nullptr);
    return cudaGetLastError();
}

cudaError_t launch_frame_to_pack64(const PackedFrame& f, uint64_t* dst, size_t dst_pitch_words, const unsigned int* err,
                                   cudaStream_t s) {
    const int rows = f.nrows(), nwords = 2 * ((f.n + 63) / 64);
    const Shape b = shape(nwords, rows, 1);
    (b.narrow ? k_words_to_pack<true> : k_words_to_pack<false>)<<<b.grid, b.block, 0, s>>>(word_origin(f), f.wpitch, rows, f.n, (uint32_t*)dst,
                                                             2 * dst_pitch_words, nwords, err);
    return cudaGetLastError();
}

cudaError_t launch_pack64_to_frame(const uint64_t* src, size_t src_pitch_words, const PackedFrame& f,
                                   GridBarrier* barrier, cudaStream_t s) {
    const int rows = f.nrows();
    const Shape b = shape(f.nw, rows, 1);
    const bool join = f.n >= 64 && f.n % 32 != 0;
    auto kernel = b.narrow ? (join ? k_pack_to_words<true, true> : k_pack_to_words<false, true>)
                           : (join ? k_pack_to_words<true, false> : k_pack_to_words<false, false>);
    kernel<<<b.grid, b.block, 0, s>>>((const uint32_t*)src, 2 * src_pitch_words, rows, f.n, word_origin(f),
                                                   f.wpitch, f.nw, barrier);
    return cudaGetLastError();
}

// --- K6: population and comparison over the inner cells -----------------------
cudaError_t launch_population(const Frame& f, unsigned long long* scratch, cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(scratch, 0, sizeof(unsigned long long), s);
    if (e != cudaSuccess) return e;
    k_population<false><<<cover((f.n + 15) / 16, f.nrows(), kRows, kReduceBlocks), kBlock, 0, s>>>(byte_rows(f),
                                                                                                  scratch);
    return cudaGetLastError();
}

cudaError_t launch_population(const PackedFrame& f, unsigned long long* scratch, cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(scratch, 0, sizeof(unsigned long long), s);
    if (e != cudaSuccess) return e;
    k_population<true><<<cover(f.nw, f.nrows(), kRows, kReduceBlocks), kBlock, 0, s>>>(word_rows(f), scratch);
    return cudaGetLastError();
}

static cudaError_t clear_compare(unsigned long long* scratch, cudaStream_t s) {
    cudaError_t e = cudaMemsetAsync(scratch, 0, sizeof(unsigned long long), s);
    if (e == cudaSuccess) e = cudaMemsetAsync(scratch + 1, 0xff, sizeof(unsigned long long), s);
    return e;
}

cudaError_t launch_compare(const Frame& f, const uint8_t* other, size_t other_pitch, unsigned long long* scratch,
                           cudaStream_t s) {
    cudaError_t e = clear_compare(scratch, s);
    if (e != cudaSuccess) return e;
    k_compare<false><<<cover((f.n + 15) / 16, f.nrows(), kRows, kReduceBlocks), kBlock, 0, s>>>(byte_rows(f), other,
                                                                                               other_pitch, scratch);
    return cudaGetLastError();
}

cudaError_t launch_compare(const PackedFrame& f, const uint8_t* other, size_t other_pitch, unsigned long long* scratch,
                           cudaStream_t s) {
    cudaError_t e = clear_compare(scratch, s);
    if (e != cudaSuccess) return e;
    k_compare<true><<<cover((f.n + 15) / 16, f.nrows(), kRows, kReduceBlocks), kBlock, 0, s>>>(word_rows(f), other,
                                                                                              other_pitch, scratch);
    return cudaGetLastError();
}

}  // namespace ltl
