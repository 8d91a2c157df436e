// k_packed.cu -- K3: bit-packed LtL step (one bit per cell).
//
// Same function as the reference's HostSolver<int> step (kezada94/CAT_cpu,
// src/CellularAutomata/Solvers/HostSolver.tpp:58-91, torus halo :93-140), with
// 32 cells per 32-bit word and the neighbour count kept bit-sliced:
//   h(row) = horizontal (2R+1)-window count of one row, as PH bit planes, by a
//            carry-save (Wallace) reduction of the 2R+1 shifted row words;
//   B      = vertical sliding sum of h over 2R+1 rows, as PB bit planes
//            (B -= h(r-R); B += h(r+R+1) while a thread walks down its band);
//   next   = s ? [smin+1 <= B <= smax+1] : [bmin <= B <= bmax]   (B includes the centre)
// evaluated with bit-sliced comparators.  Every operation acts on 32 cells.
#include <algorithm>

#include "packed_core.cuh"

namespace ltl {

constexpr int kPackedWarps = 4;

// Rows per work item when no tuned value applies: as few bands as fill every
// resident warp once (each band re-counts 2R+1 rows to start its window, so
// fewer, longer bands waste less), split further only where a band would be
// longer than 256 rows.
static int packed_band_rows(int n, int n_wstrips, int resident_warps) {
    const int per_wave = std::max(1, resident_warps / std::max(n_wstrips, 1));
    int bands = per_wave;
    while ((n + bands - 1) / bands > 256) bands += per_wave;
    return std::max(16, (n + bands - 1) / bands);
}

template <int R, bool FUSE>
__global__ void __launch_bounds__(kPackedWarps * 32)
k_packed_step(const uint32_t* __restrict__ cur, uint32_t* __restrict__ nxt, int rows, int nw, int HR, int HW,
              size_t wp, int n_wstrips, int n_items, int band_rows, const __grid_constant__ PackedRule pr) {
    using Ring = PackedRing<R, kPackedWarps>;
    extern __shared__ uint32_t ring_all[];
    const int lane = threadIdx.x & 31;
    const int wid = threadIdx.x >> 5;
    uint32_t* ring_lane = ring_all + (size_t)wid * Ring::WARP_WORDS + lane;
    const int gwarp = blockIdx.x * kPackedWarps + wid;
    const int gwarps = gridDim.x * kPackedWarps;

    for (int item = gwarp; item < n_items; item += gwarps) {
        const int ws = item % n_wstrips;
        const int band = item / n_wstrips;
        const int r0 = band * band_rows;
        const int r1 = min(r0 + band_rows, rows);
        const int w = ws * 32 + lane;     // inner word
        const bool active = w <= nw;      // w == nw is the right halo word (neighbour of the last word)
        const bool outputs = w < nw;
        packed_band<R, Ring::fits, FUSE>(cur, nxt, wp, HR, r0, r1, HW + w, active, outputs, lane, ring_lane, pr,
                                         rows, nw);
        __syncwarp();
    }
}

bool packed_supported(int n, int radius) { return radius >= 1 && radius <= 32 && n >= radius; }

// The step writes the output frame's halo itself (packed_band's kFuse) where
// every halo word is a whole inner word: n a multiple of 32, one halo word.
bool packed_fused_halo(const PackedFrame& f, int radius) {
    return f.HW == 1 && f.n % 32 == 0 && f.n >= 64 && f.nrows() >= 2 * radius + 2;
}

template <int R>
static cudaError_t launch_packed_r(const PackedFrame& c, const PackedFrame& x, const PackedRule& pr,
                                   int band_override, cudaStream_t s) {
    int dev = 0, sms = 148, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    // strips of 32 words cover the inner words; a lane whose word is the right
    // halo word (w == nw) only feeds its left neighbour, and lane 31 loads the
    // word past its own directly, so no strip is needed for the halo alone
    const int n_wstrips = (c.nw + 31) / 32;
    const int smem = PackedRing<R, kPackedWarps>::fits ? PackedRing<R, kPackedWarps>::BYTES : 0;
    const bool fuse = packed_fused_halo(x, R);
    auto kernel = fuse ? k_packed_step<R, true> : k_packed_step<R, false>;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kPackedWarps * 32, smem);
    if (per_sm < 1) per_sm = 1;
    const int band_rows =
        band_override > 0 ? band_override : packed_band_rows(c.nrows(), n_wstrips, sms * per_sm * kPackedWarps);
    const int bands = (c.nrows() + band_rows - 1) / band_rows;
    const int items = n_wstrips * bands;
    int ctas = std::min((items + kPackedWarps - 1) / kPackedWarps, sms * per_sm);
    kernel<<<ctas, kPackedWarps * 32, smem, s>>>(c.words, x.words, c.nrows(), c.nw, c.HR, c.HW, c.wpitch,
                                                           n_wstrips, items, band_rows, pr);
    return cudaGetLastError();
}

template <int R>
static cudaError_t prepare_packed_r() {
    const int smem = PackedRing<R, kPackedWarps>::fits ? PackedRing<R, kPackedWarps>::BYTES : 0;
    if (smem <= 48 * 1024) return cudaSuccess;
    cudaError_t e = cudaFuncSetAttribute(k_packed_step<R, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(k_packed_step<R, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
}

cudaError_t packed_prepare(int radius) {
    switch (radius) {
#define LTL_PP(r) \
    case r: return prepare_packed_r<r>();
        LTL_PP(1) LTL_PP(2) LTL_PP(3) LTL_PP(4) LTL_PP(5) LTL_PP(6) LTL_PP(7) LTL_PP(8)
        LTL_PP(9) LTL_PP(10) LTL_PP(11) LTL_PP(12) LTL_PP(13) LTL_PP(14) LTL_PP(15) LTL_PP(16)
        LTL_PP(17) LTL_PP(18) LTL_PP(19) LTL_PP(20) LTL_PP(21) LTL_PP(22) LTL_PP(23) LTL_PP(24)
        LTL_PP(25) LTL_PP(26) LTL_PP(27) LTL_PP(28) LTL_PP(29) LTL_PP(30) LTL_PP(31) LTL_PP(32)
#undef LTL_PP
        default: return cudaSuccess;
    }
}

cudaError_t launch_packed_step(const PackedFrame& cur, const PackedFrame& nxt, const Rule& rule, int band_rows,
                               cudaStream_t s) {
    PackedRule pr = make_packed_rule(rule);
    switch (rule.radius) {
#define LTL_PR(r) \
    case r: return launch_packed_r<r>(cur, nxt, pr, band_rows, s);
        LTL_PR(1) LTL_PR(2) LTL_PR(3) LTL_PR(4) LTL_PR(5) LTL_PR(6) LTL_PR(7) LTL_PR(8)
        LTL_PR(9) LTL_PR(10) LTL_PR(11) LTL_PR(12) LTL_PR(13) LTL_PR(14) LTL_PR(15) LTL_PR(16)
        LTL_PR(17) LTL_PR(18) LTL_PR(19) LTL_PR(20) LTL_PR(21) LTL_PR(22) LTL_PR(23) LTL_PR(24)
        LTL_PR(25) LTL_PR(26) LTL_PR(27) LTL_PR(28) LTL_PR(29) LTL_PR(30) LTL_PR(31) LTL_PR(32)
#undef LTL_PR
        default: return cudaErrorInvalidValue;
    }
}

// ---------------------------------------------------------------------------
// Packed halo: column halo bits of inner rows (bit position p of the frame row
// holds cell (p - 32*HW) mod n), then whole top/bottom rows copied from the
// inner rows they wrap to.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t packed_bit(const uint32_t* row, int HW, int cell) {
    int p = 32 * HW + cell;
    return (row[p >> 5] >> (p & 31)) & 1u;
}

__global__ void k_packed_halo_cols(uint32_t* __restrict__ g, int n, int rows, int nw, int HR, int HW, size_t wp) {
    // per inner row: words [0, HW) and [HW + nw - 1, HW + nw + HW)
    const int per_row = 2 * HW + 1;
    const long long total = (long long)rows * per_row;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
         t += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(t / per_row);
        const int k = (int)(t % per_row);
        const int fw = k < HW ? k : HW + nw - 1 + (k - HW);
        uint32_t* row = g + (size_t)(HR + i) * wp;
        auto slow = [&]() -> uint32_t {
            uint32_t v = 0u;
            if (fw == HW + nw - 1) {
                // last inner word: keep its inner bits, rewrite the bits past n
                const int inner_bits = n - 32 * (nw - 1);
                v = inner_bits >= 32 ? row[fw] : (row[fw] & ((1u << inner_bits) - 1u));
                for (int b = inner_bits; b < 32; ++b) {
                    int cell = 32 * (nw - 1) + b;
                    v |= packed_bit(row, HW, cell % n) << b;
                }
            } else {
                for (int b = 0; b < 32; ++b) {
                    int cell = 32 * (fw - HW) + b;
                    int src = ((cell % n) + n) % n;
                    v |= packed_bit(row, HW, src) << b;
                }
            }
            return v;
        };
        const uint32_t v = HW == 1 ? packed_halo_word(row, fw, n, nw, slow) : slow();
        // the halo words only read inner bits (< n), never bits written here
        row[fw] = v;
    }
}

__global__ void k_packed_halo_rows(uint32_t* __restrict__ g, int rows, int HR, size_t wp) {
    const int band = blockIdx.y;  // 0 .. 2HR-1
    const int r = band < HR ? band : rows + band;
    const int src = HR + (((r - HR) % rows) + rows) % rows;
    uint32_t* d = g + (size_t)r * wp;
    const uint32_t* sp = g + (size_t)src * wp;
    for (int w = blockIdx.x * blockDim.x + threadIdx.x; w < (int)wp; w += gridDim.x * blockDim.x) d[w] = sp[w];
}

cudaError_t launch_packed_halo(const PackedFrame& f, cudaStream_t s) {
    const long long total = (long long)f.nrows() * (2 * f.HW + 1);
    int blocks = (int)std::min<long long>((total + 127) / 128, 4096);
    k_packed_halo_cols<<<blocks, 128, 0, s>>>(f.words, f.n, f.nrows(), f.nw, f.HR, f.HW, f.wpitch);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    dim3 g2((unsigned)std::max<size_t>(1, std::min<size_t>((f.wpitch + 127) / 128, 64)), (unsigned)(2 * f.HR));
    k_packed_halo_rows<<<g2, 128, 0, s>>>(f.words, f.nrows(), f.HR, f.wpitch);
    return cudaGetLastError();
}

}  // namespace ltl
