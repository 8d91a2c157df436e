// transfer_core.cuh -- byte cells <-> bits, 16 cells at a time, shared by the
// transfer kernels of single grids (k_transfer.cu) and batches (k_batch.cu).
#pragma once

#include <cstdint>

namespace ltl {

// Four 0/1 bytes of a word -> 4 bits: the multiply places byte k's bit at bit
// 24 + k with no two partial products overlapping (so no carries), and back:
// the 4 bits of a nibble spread to bit 0 of each byte by copies 7 bits apart.
__device__ __forceinline__ uint32_t bytes4_to_bits(uint32_t w) { return ((w & 0x01010101u) * 0x01020408u) >> 24; }
__device__ __forceinline__ uint32_t bits4_to_bytes(uint32_t nib) { return (nib * 0x00204081u) & 0x01010101u; }

// Per byte: 1 if the byte is not zero (7-bit add, the top bit joined in: no
// carry leaves a byte).
__device__ __forceinline__ uint32_t nonzero4(uint32_t w) {
    return ((((w & 0x7f7f7f7fu) + 0x7f7f7f7fu) | w) >> 7) & 0x01010101u;
}

template <bool kNonzero>
__device__ __forceinline__ uint32_t cells16_to_bits(uint4 v) {
    uint32_t q[4] = {v.x, v.y, v.z, v.w};
    uint32_t r = 0u;
#pragma unroll
    for (int k = 0; k < 4; ++k) r |= bytes4_to_bits(kNonzero ? nonzero4(q[k]) : q[k]) << (4 * k);
    return r;
}

__device__ __forceinline__ uint4 bits16_to_cells(uint32_t b) {
    return make_uint4(bits4_to_bytes(b & 15u), bits4_to_bytes((b >> 4) & 15u), bits4_to_bytes((b >> 8) & 15u),
                      bits4_to_bytes((b >> 12) & 15u));
}

// The 16 bytes at p, of a buffer whose bytes are [lo, hi).  Bytes outside the
// buffer come back as 0 and are not read.  p may have any alignment.  kStream: whole
// vectors are marked to be evicted first (so are store16's): cells that become words,
// or come from them, pass through once and would push the words out of L2 (16384^2
// cells to words and back 136 us without marks or with those of the stores alone, 107
// with both; compare 147 / 123).  A copy of cells is slower with them, 84 / 96.
template <bool kStream>
__device__ __forceinline__ uint4 load16(const uint8_t* p, const uint8_t* lo, const uint8_t* hi) {
    const uintptr_t a = (uintptr_t)p;
    if ((a & 15) == 0 && p >= lo && p + 16 <= hi) return kStream ? __ldcs((const uint4*)p) : *(const uint4*)p;
    const uint32_t* q = (const uint32_t*)(a & ~(uintptr_t)3);
    const int sh = 8 * (int)(a & 3);
    if ((const uint8_t*)q >= lo && (const uint8_t*)(q + 5) <= hi) {
        const uint32_t w0 = q[0], w1 = q[1], w2 = q[2], w3 = q[3], w4 = sh ? q[4] : 0u;
        return make_uint4(__funnelshift_r(w0, w1, sh), __funnelshift_r(w1, w2, sh), __funnelshift_r(w2, w3, sh),
                          __funnelshift_r(w3, w4, sh));
    }
    uint32_t r[4] = {0u, 0u, 0u, 0u};
#pragma unroll
    for (int k = 0; k < 16; ++k)
        if (p + k >= lo && p + k < hi) r[k >> 2] |= (uint32_t)p[k] << (8 * (k & 3));
    return make_uint4(r[0], r[1], r[2], r[3]);
}

// Bytes [from, to) of v to dst .. dst + 15 (dst 16-byte aligned; a whole vector
// where from = 0 and to = 16).
template <bool kStream>
__device__ __forceinline__ void store16(uint8_t* dst, uint4 v, int from, int to) {
    if (from <= 0 && to >= 16) {
        if constexpr (kStream) __stcs((uint4*)dst, v);
        else *(uint4*)dst = v;
        return;
    }
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int k = 0; k < 16; ++k)
        if (k >= from && k < to) dst[k] = (uint8_t)(w[k >> 2] >> (8 * (k & 3)));
}

// 16 bits of a word row from bit c on (c may be negative down to -15: those
// bits are 0), the row holding `nwords` words.
__device__ __forceinline__ uint32_t bits16_at(const uint32_t* row, int c, int nwords) {
    const int w = c >> 5;  // floor
    const uint32_t lo = w >= 0 && w < nwords ? __ldg(row + w) : 0u;
    const uint32_t hi = (c & 31) > 16 && w + 1 < nwords ? __ldg(row + w + 1) : 0u;
    return __funnelshift_r(lo, hi, c & 31) & 0xffffu;
}

// Items `at`, at + stride, .. of an array of `width` items per row, in row-major order,
// as rows and columns.  No item number is formed: the number of 16-cell vectors of a
// grid passes 2^31 at 185,352 cells a side, that of its words at 262,144.
struct RowWalk {
    int row, col;
    int width, rows_on, cols_on;  // what a stride moves
    __host__ __device__ RowWalk(int at, int stride, int width_)
        : row(at / width_), col(at % width_), width(width_), rows_on(stride / width_), cols_on(stride % width_) {}
    __host__ __device__ void next() {
        row += rows_on;
        col += cols_on;
        if (col >= width) {
            col -= width;
            ++row;
        }
    }
};

// Byte offset of the first 16-byte vector of a destination row relative to its
// first cell: 0 if aligned, else negative (that vector starts before the row).
__device__ __forceinline__ int lead(const uint8_t* p) { return -(int)((uintptr_t)p & 15); }

}  // namespace ltl
