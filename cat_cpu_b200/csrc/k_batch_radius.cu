// k_batch_radius.cu -- K4, per-generation mode: the kernels of one radius (LTL_RADIUS;
// build.py compiles a part for each, see batch_ops.h).
#include <algorithm>

#include "batch_ops.h"
#include "packed_core.cuh"

namespace ltl {

// ---------------------------------------------------------------------------
// Per-step kernel for the streamed grids of one rule class.
// ---------------------------------------------------------------------------
// The walk in the form that a side needs, one word per lane.
template <int R, bool kRing, bool kConst>
__device__ __forceinline__ void batch_walk(const uint32_t* cur, uint32_t* nxt, const BatchGrid& g, int r0, int r1,
                                           int w0, uint32_t* ring, int lane, const PackedRule& pr) {
    if (g.n < 64)
        packed_walk<R, 1, kRing, kEdgeTiny, kConst>(cur, nxt, g.wp, g.n, g.nw, g.n, r0, r1, w0, ring, lane, pr);
    else if (g.n % 32 == 0)
        packed_walk<R, 1, kRing, kEdgeNone, kConst>(cur, nxt, g.wp, g.n, g.nw, g.n, r0, r1, w0, ring, lane, pr);
    else
        packed_walk<R, 1, kRing, kEdgeRagged, kConst>(cur, nxt, g.wp, g.n, g.nw, g.n, r0, r1, w0, ring, lane, pr);
}

template <int R>
__global__ void __launch_bounds__(kBatchWarps * 32)
k_batch_step(const uint32_t* __restrict__ cur, uint32_t* __restrict__ nxt, const BatchGrid* __restrict__ grids,
             const int4* __restrict__ items, int n_items, const __grid_constant__ PackedRule pr) {
    extern __shared__ __align__(16) uint32_t ring_all[];
    const int lane = threadIdx.x & 31;
    const int wid = threadIdx.x >> 5;
    uint32_t* ring = ring_all + (size_t)wid * PackedRing<R, 1>::WARP_WORDS;
    const int gwarp = blockIdx.x * kBatchWarps + wid;
    const int gwarps = gridDim.x * kBatchWarps;
    for (int it = gwarp; it < n_items; it += gwarps) {
        const int4 item = items[it];  // grid, r0, r1, word strip
        const BatchGrid g = grids[item.x];
        const int w = item.w * 32 + lane;
        if (w < g.nw) batch_walk<R, true, true>(cur + g.off, nxt + g.off, g, item.y, item.z, w, ring, lane, pr);
    }
}

// ---------------------------------------------------------------------------
// Resident kernel: whole grids in shared memory for `steps` generations.  The
// leaving row is counted again (shared memory holds the two grids, no rings).
// ---------------------------------------------------------------------------
template <int R>
__global__ void __launch_bounds__(kResThreads, 1)
k_batch_resident(const uint32_t* __restrict__ src, uint32_t* __restrict__ dst, const BatchGrid* __restrict__ grids,
                 const int* __restrict__ list, int n_list, int steps, const __grid_constant__ PackedRule pr) {
    extern __shared__ __align__(16) uint32_t sm[];
    for (int li = blockIdx.x; li < n_list; li += gridDim.x) {
        const BatchGrid g = grids[list[li]];
        const int words = g.n * g.wp;
        uint32_t* bufA = sm;
        uint32_t* bufB = sm + words;
        for (int t = threadIdx.x; t < words; t += blockDim.x) bufA[t] = src[g.off + t];
        __syncthreads();
        const int bands = min(g.n, max(1, (int)blockDim.x / g.nw));
        const int band_rows = (g.n + bands - 1) / bands;
        for (int s = 0; s < steps; ++s) {
            for (int it = threadIdx.x; it < g.nw * bands; it += blockDim.x) {
                const int band = it / g.nw, r0 = band * band_rows, r1 = min(r0 + band_rows, g.n);
                if (r0 < r1) batch_walk<R, false, false>(bufA, bufB, g, r0, r1, it - band * g.nw, nullptr, 0, pr);
            }
            __syncthreads();
            uint32_t* t = bufA;
            bufA = bufB;
            bufB = t;
        }
        for (int t = threadIdx.x; t < words; t += blockDim.x) dst[g.off + t] = bufA[t];
        __syncthreads();
    }
}

template <int R>
cudaError_t BatchOps<R>::step(const uint32_t* cur, uint32_t* nxt, const BatchGrid* grids, const int4* items,
                              int n_items, const PackedRule& pr, int sms, cudaStream_t s) {
    const int smem = kBatchWarps * PackedRing<R, 1>::WARP_WORDS * 4;
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_batch_step<R>, kBatchWarps * 32, smem);
    if (per_sm < 1) per_sm = 1;
    const int ctas = std::max(1, std::min((n_items + kBatchWarps - 1) / kBatchWarps, sms * per_sm));
    k_batch_step<R><<<ctas, kBatchWarps * 32, smem, s>>>(cur, nxt, grids, items, n_items, pr);
    return cudaGetLastError();
}

// Shared-memory limit of the streamed step kernel (its h ring), set once per
// radius outside any stream capture.
template <int R>
cudaError_t BatchOps<R>::prepare_step() {
    return cudaFuncSetAttribute(k_batch_step<R>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                kBatchWarps * PackedRing<R, 1>::WARP_WORDS * 4);
}

template <int R>
cudaError_t BatchOps<R>::resident(const uint32_t* src, uint32_t* dst, const BatchGrid* grids, const int* list,
                                  int n_list, int steps, const PackedRule& pr, size_t smem, int sms, cudaStream_t s) {
    const int ctas = std::max(1, std::min(n_list, sms));
    k_batch_resident<R><<<ctas, kResThreads, smem, s>>>(src, dst, grids, list, n_list, steps, pr);
    return cudaGetLastError();
}

template <int R>
cudaError_t BatchOps<R>::prepare_resident() {
    return cudaFuncSetAttribute(k_batch_resident<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, kResSmemLimit);
}

#ifdef LTL_RADIUS
template struct BatchOps<LTL_RADIUS>;
#else
#define LTL_ALL(r) template struct BatchOps<r>;
LTL_BATCH_RADII(LTL_ALL)
#undef LTL_ALL
#endif

}  // namespace ltl
