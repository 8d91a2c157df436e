// ltl_internal.cuh -- shared layout, rule and error helpers of libltl_b200.
//
// Device grid layout (every variant that stores one byte per cell):
//   a frame of (n + 2H) rows, `pitch` bytes per row, inner cell (i, j) at
//   base[(H + i) * pitch + H + j].  H is a multiple of 16 and >= R * depth, the
//   halo holds torus copies of inner cells (frame cell (r, c) = inner
//   ((r - H) mod n, (c - H) mod n)), refreshed by k_halo_fill before each pass.
//   This is the reference's CADataDomain layout (CADataDomain.tpp:4-98, inner
//   (i,j) at (i+h)*(n+2h) + j+h) with the halo rounded up to 16 bytes and the
//   pitch padded so that 16-byte vector and TMA accesses stay aligned and a
//   16-byte load that starts inside the right halo stays inside its row.
#pragma once

#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

namespace ltl {

constexpr int kWarp = 32;

struct Frame {
    uint8_t* base;   // frame origin (row 0, column 0)
    int n;           // inner columns (and rows, unless `rows` is set)
    int H;           // halo width (cells)
    size_t pitch;    // bytes per frame row
    int rows = 0;    // inner rows of a rectangular torus (0: square, n rows)
    __host__ __device__ int nrows() const { return rows ? rows : n; }
    __host__ __device__ uint8_t* inner(int i, int j) const { return base + (size_t)(H + i) * pitch + H + j; }
    __host__ __device__ const uint8_t* cinner(int i, int j) const {
        return base + (size_t)(H + i) * pitch + H + j;
    }
};

__host__ __device__ inline size_t round_up(size_t v, size_t m) { return (v + m - 1) / m * m; }

inline int halo_for(int radius, int depth) {
    int h = radius * depth;
    if (h < 16) h = 16;
    return (int)round_up((size_t)h, 16);
}

inline size_t pitch_for(int n, int H) { return round_up((size_t)n + 2 * (size_t)H + 16, 64); }

// Rule in the reference's centre-excluded convention.
struct Rule {
    int radius, smin, smax, bmin, bmax;
};

// Thresholds on the box count B (centre INCLUDED) for 8-bit SWAR lanes holding
// B <= 127: alive cell survives iff slo <= B <= shi (slo = smin+1, shi = smax+1,
// since k = B - 1), dead cell is born iff blo <= B <= bhi.  Empty intervals are
// encoded lo = 128, hi = 0; lo is clamped to [0,128], hi to [0,127].  Each value
// is broadcast to the four byte lanes, lo as 0x80 - lo (so that B + (0x80 - lo)
// has bit 7 set iff B >= lo, without a carry into the next lane) and hi with
// the 0x80 marker bit (0x80 + hi - B has bit 7 set iff B <= hi).  `d*` hold the
// live value minus the dead one of a single lane: a multiply-add of the centres
// (0/1 lanes) selects for all four lanes at once, on the FMA pipe that the rest of
// the step leaves idle.  Every selected lane value is in [0, 0xff], so the sum over
// lanes is exact whatever the sign of d.  16384^2 R = 5, two generations per pass,
// with the selects as XOR and AND on the ALU 83.5 us per generation, so 78.0.
struct RuleSwar8 {
    uint32_t nlo0, hiH0;  // dead cell (birth interval)
    uint32_t dnlo, dhiH;  // live-cell (survival) minus dead-cell value of one lane, mod 2^32
};

inline void clamp_interval8(int lo, int hi, uint32_t& nlo_out, uint32_t& hi_out) {
    if (lo < 0) lo = 0;
    if (hi > 127) hi = 127;
    if (hi < lo || lo > 127) {
        lo = 128;
        hi = 0;
    }
    nlo_out = (uint32_t)(0x80 - lo);
    hi_out = (uint32_t)hi | 0x80u;
}

inline RuleSwar8 make_rule_swar8(const Rule& r) {
    uint32_t nlo0, hi0, nlo1, hi1;
    clamp_interval8(r.bmin, r.bmax, nlo0, hi0);
    clamp_interval8(r.smin + 1, r.smax + 1, nlo1, hi1);
    return RuleSwar8{nlo0 * 0x01010101u, hi0 * 0x01010101u, nlo1 - nlo0, hi1 - hi0};
}

// Per byte lane: 1 if the lane's cell is alive in the next generation.
// B: four box counts (centre included, each <= 127); s: four centre cells (0/1).
__device__ __forceinline__ uint32_t rule_swar8(uint32_t B, uint32_t s, const RuleSwar8& q) {
    const uint32_t ge = B + (s * q.dnlo + q.nlo0);    // bit 7 set iff B >= lo
    const uint32_t le = (s * q.dhiH + q.hiH0) - B;    // bit 7 set iff hi >= B
    return (ge & le & 0x80808080u) >> 7;
}

__device__ __forceinline__ int rule_scalar(int k, int s, int smin, int smax, int bmin, int bmax) {
    return s ? (k >= smin && k <= smax) : (k >= bmin && k <= bmax);
}

__device__ __forceinline__ int wrap_mod(int v, int n) {
    int r = v % n;
    return r < 0 ? r + n : r;
}

#ifdef __CUDACC__
// Chained launches: a step's kernel may be put on the SMs while the one before it in the
// stream still runs its last CTAs, and waits there for that one's end (chain_wait, before
// anything of the grid is touched).  Hides the launch and the prologue behind the tail.
// For kernels of one CTA per SM: the tensor step at 8192^2 R = 5 33.5 -> 32.0 us, 16384^2
// 115.4 -> 114.3 (30.3 and 108.2 since it waits after its prologue's block barrier).  Where several CTAs share an SM the early ones crowd the SMs that are
// done first, and the step is as long as the fullest SM (band walk 16384^2 R = 2 31 ->
// 43 us, plain R = 64 6001^2 39 -> 50), so those kernels are launched plainly.
template <class... P, class... A>
inline cudaError_t launch_chained(void (*kernel)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                                  A... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

__device__ __forceinline__ void chain_wait() {
    asm volatile("griddepcontrol.launch_dependents;");
    asm volatile("griddepcontrol.wait;" ::: "memory");
}
#endif

}  // namespace ltl

// Host-side error reporting (ltl_abi.cu).
void ltl_set_error(const char* fmt, ...);
