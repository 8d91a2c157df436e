// k_batch.cu -- K4: many independent tori of uneven size, radius and rule,
// advanced together (ltl_batch_* in include/ltl.h).
//
// Semantics per grid are the reference's HostSolver<int> step (kezada94/CAT_cpu,
// src/CellularAutomata/Solvers/HostSolver.tpp:58-140); the reference runs one
// grid per process (CPUBenchmark.cpp:63-85).  Design:
//   - every grid is stored bit-packed (packed_core.cuh) in one device arena,
//     two arenas ping-pong; no form has a halo, the walk wraps rows and words in
//     its loads;
//   - persistent mode (the default): one launch runs every generation of every
//     grid of a call (k_batch_persist below);
//   - per-generation mode (k_batch_radius.cu): grids are grouped into rule classes
//     (radius + rule), each a kernel instantiation with its masks in the constant
//     bank.  "Resident" grids, whose two packed copies fit in one SM's shared memory,
//     are advanced all steps of a call in one launch; the others one generation per
//     launch over a (grid, row band, word strip) work list, with the resident
//     launches beside them on a forked stream;
//   - either way a call is a CUDA graph, made for its step count and starting arena.
#include <algorithm>
#include <cstring>
#include <map>
#include <new>
#include <vector>

#include "../../include/ltl.h"
#include "batch_ops.h"
#include "batch_split.h"
#include "grid_barrier.cuh"
#include "packed_core.cuh"
#include "transfer_core.cuh"

namespace ltl {

// ---------------------------------------------------------------------------
// Persistent kernel: one launch advances every grid of the batch through all the
// generations of one ltl_batch_step.  Grids whose share of the work is more than
// one CTA's get a group of CTAs each (batch_split decides; a group barrier between
// generations, so the launch is cooperative); when its group is done, and from the
// start where it has none, a CTA takes whole grids from a device counter, the most
// work first, with only CTA barriers between generations.  A grid stays in L1 and
// L2 for the whole run, and no per-generation launch is made.
//
// A CTA is four warps (one per scheduler) and walks long bands; several CTAs per SM
// on different grids fill the ALU and cover each other's barriers.  The band walk
// has two words per lane up to R = 5 and lanes numbered over
// (band, word group), so none idles on narrow rows.  Bound by the ALU where there are
// many grids (512 grids of R <= 2: 6340 GCUPS), by barriers and band starts where
// there are few.  256 generations of 64 and of 1024 grids of sides 64..2048, R 1..8
// (without transfers): 52 and 70 ms with one CTA of eight warps per grid, 3.8 and
// 42 ms so.
// ---------------------------------------------------------------------------
// A CTA's first task: its rank in the group of grid `grid` (size 0: none).
struct BatchGroup {
    int grid, rank, size;
};

// The groups' barriers (one per grid), the word set if a wait runs out, the waits' limit.
struct BatchWaits {
    GridBarrier* barriers;
    unsigned int* err;
    BarrierLimit limit;
};

// Not inlined: forms and radii that share one function share its registers (255, and
// spills in the walk's loop).  One by one they are held to the 128 that four CTAs per SM
// leave, at 20 to 100 bytes of spills in most, and are faster so (168 registers and three
// CTAs: 48.6 ms against 42.2 for the 1024-grid ensemble).
template <int R, int W, int EDGE>
__device__ __noinline__ bool persist_form(const BatchGrid& g, uint32_t* f0, uint32_t* f1, int steps, int rank,
                                          int size, const BatchWaits& waits, int grid, const PackedRule& rule,
                                          uint32_t* ring) {
    const PackedRule pr = rule;  // the masks the comparators use: loaded once, as far as registers go
    GridBarrierWait group(waits.barriers + grid, size, waits.limit);
    const int lanes = size * kPersistThreads, id = rank * kPersistThreads + threadIdx.x;
    const int groups = (g.nw + W - 1) / W;
    const int bands = min(g.n, max(1, lanes / groups));
    const int band_rows = (g.n + bands - 1) / bands;
    const int items = groups * ((g.n + band_rows - 1) / band_rows);
    for (int s = 0; s < steps; ++s) {
        const uint32_t* src = (s & 1) ? f1 : f0;
        uint32_t* dst = (s & 1) ? f0 : f1;
        for (int it = id; it < items; it += lanes) {
            const int band = it / groups, r0 = band * band_rows;
            packed_walk<R, W, true, EDGE, false>(src, dst, g.wp, g.n, g.nw, g.n, r0, min(r0 + band_rows, g.n),
                                                 W * (it - band * groups), ring, threadIdx.x & 31, pr);
        }
        if (!group.wait(waits.err)) return false;
    }
    return true;
}

// All generations of one grid (radius R) by this CTA, or its part of them.
template <int R>
__device__ __forceinline__ bool persist_grid(const BatchGrid& g, uint32_t* a0, uint32_t* a1, int steps, int rank, int size,
                             const BatchWaits& waits, int grid, const PackedRule& rule, uint32_t* ring_all) {
    constexpr int W = persist_words(R);
    uint32_t* ring = ring_all + (threadIdx.x >> 5) * PackedRing<R, W>::WARP_WORDS;
    uint32_t* f0 = a0 + g.off;
    uint32_t* f1 = a1 + g.off;
    if (!packed_two_words(g.n)) return persist_form<R, 1, kEdgeTiny>(g, f0, f1, steps, rank, size, waits, grid, rule, ring);
    if (packed_edge(g.n, W) == kEdgeNone)
        return persist_form<R, W, kEdgeNone>(g, f0, f1, steps, rank, size, waits, grid, rule, ring);
    return persist_form<R, W, kEdgeRagged>(g, f0, f1, steps, rank, size, waits, grid, rule, ring);
}

__global__ void __launch_bounds__(kPersistThreads, 4)
k_batch_persist(uint32_t* a0, uint32_t* a1, const BatchGrid* __restrict__ grids, const PackedRule* __restrict__ rules,
                const BatchGroup* __restrict__ first, const __grid_constant__ BatchWaits waits,
                const int* __restrict__ order, int n_order, int* next, int steps) {
    extern __shared__ __align__(16) uint32_t ring_all[];
    __shared__ int s_item;
    BatchGroup task = first[blockIdx.x];
    while (true) {
        if (task.size == 0) {
            if (threadIdx.x == 0) s_item = atomicAdd(next, 1);
            __syncthreads();
            const int li = s_item;
            __syncthreads();  // every thread has read s_item before it is overwritten
            if (li >= n_order) break;
            task = BatchGroup{order[li], 0, 1};
        }
        const BatchGrid g = grids[task.grid];
        bool ok = true;
        switch (g.R) {
#define LTL_C(r)                                                                                                    \
    case r:                                                                                                         \
        ok = persist_grid<r>(g, a0, a1, steps, task.rank, task.size, waits, task.grid, rules[g.cls],       \
                             ring_all);                                                                             \
        break;
            LTL_BATCH_RADII(LTL_C)
#undef LTL_C
            default: break;
        }
        if (!ok) break;
        task.size = 0;
    }
}

// Shared memory of the persistent kernel for a batch whose largest radius is R:
// its warps' rings of window counts.
template <int R>
static size_t persist_ring_bytes() {
    return (size_t)kPersistWarps * PackedRing<R, persist_words(R)>::WARP_WORDS * 4;
}

// ---------------------------------------------------------------------------
// Dense staging <-> arena (all grids of a list, or one grid)
// ---------------------------------------------------------------------------
// (memory-bound like k_transfer.cu's kernels: 16-byte vectors of cells.  A grid's
// rows are n bytes apart in the staging buffer, so most rows start unaligned.)
__global__ void k_batch_pack(const uint8_t* __restrict__ cells, uint32_t* __restrict__ arena,
                             const BatchGrid* __restrict__ grids, int first, GridBarrier* barriers) {
    const BatchGrid g = grids[first + blockIdx.y];
    // (a group whose wait ran out leaves its barrier at some count in between)
    if (blockIdx.x == 0 && threadIdx.x == 0) barriers[first + blockIdx.y].arrived = 0;
    const uint8_t* c = cells + g.cell_off;
    const uint8_t* end = c + (size_t)g.n * g.n;
    const int at = blockIdx.x * blockDim.x + threadIdx.x;
    if (at >= (long long)g.n * g.nw) return;  // (most threads of a small grid: before the walk's divisions)
    for (RowWalk t(at, gridDim.x * blockDim.x, g.nw); t.row < g.n; t.next()) {
        const int i = t.row, w = t.col;
        const uint8_t* p = c + (size_t)i * g.n + 32 * w;
        const int valid = g.n - 32 * w;
        uint32_t v = cells16_to_bits<true>(load16<true>(p, c, end));
        if (valid > 16) v |= cells16_to_bits<true>(load16<true>(p + 16, c, end)) << 16;
        if (valid < 32) {
            v &= (1u << valid) - 1u;
            if (g.n >= 64) {
                const uint8_t* q = c + (size_t)i * g.n;
                v = join_word(v, cells16_to_bits<true>(load16<true>(q, c, end)) |
                                     (cells16_to_bits<true>(load16<true>(q + 16, c, end)) << 16), g.n);
            }
        }
        arena[g.off + (size_t)i * g.wp + w] = v;
    }
}

__global__ void k_batch_unpack(const uint32_t* __restrict__ arena, uint8_t* __restrict__ cells,
                               const BatchGrid* __restrict__ grids, int first) {
    const BatchGrid g = grids[first + blockIdx.y];
    uint8_t* dst = cells + g.cell_off;
    const int vecs = (g.n + 15) / 16 + 1;  // aligned vectors a row may touch
    const int at = blockIdx.x * blockDim.x + threadIdx.x;
    if (at >= (long long)g.n * vecs) return;
    for (RowWalk t(at, gridDim.x * blockDim.x, vecs); t.row < g.n; t.next()) {
        const int i = t.row;
        uint8_t* row = dst + (size_t)i * g.n;
        const int c = lead(row) + 16 * t.col;
        if (c >= g.n) continue;
        const uint32_t bits = bits16_at(arena + g.off + (size_t)i * g.wp, c, g.nw);
        store16<true>(row + c, bits16_to_cells(bits), -c, g.n - c);
    }
}

// ---------------------------------------------------------------------------
// Launch helpers per radius (R <= 32 in the packed representation)
// ---------------------------------------------------------------------------
template <int R>
static size_t res_smem_bytes(int n) {
    const int nw = (n + 31) / 32;
    const int wp = (nw + 3) / 4 * 4;
    return 2ull * (size_t)n * wp * 4;
}

static cudaError_t batch_step_dispatch(int R, const uint32_t* cur, uint32_t* nxt, const BatchGrid* grids,
                                       const int4* items, int n_items, const PackedRule& pr, int sms, cudaStream_t s) {
    switch (R) {
#define LTL_C(r) \
    case r: return BatchOps<r>::step(cur, nxt, grids, items, n_items, pr, sms, s);
        LTL_BATCH_RADII(LTL_C)
#undef LTL_C
        default: return cudaErrorInvalidValue;
    }
}

static cudaError_t batch_resident_dispatch(int R, const uint32_t* src, uint32_t* dst, const BatchGrid* grids,
                                           const int* list, int n_list, int steps, const PackedRule& pr, size_t smem,
                                           int sms, cudaStream_t s) {
    switch (R) {
#define LTL_C(r) \
    case r: return BatchOps<r>::resident(src, dst, grids, list, n_list, steps, pr, smem, sms, s);
        LTL_BATCH_RADII(LTL_C)
#undef LTL_C
        default: return cudaErrorInvalidValue;
    }
}

static cudaError_t batch_step_prepare_dispatch(int R) {
    switch (R) {
#define LTL_BSP(r) \
    case r: return BatchOps<r>::prepare_step();
        LTL_BATCH_RADII(LTL_BSP)
#undef LTL_BSP
        default: return cudaErrorInvalidValue;
    }
}

static cudaError_t batch_prepare_dispatch(int R) {
    switch (R) {
#define LTL_C(r) \
    case r: return BatchOps<r>::prepare_resident();
        LTL_BATCH_RADII(LTL_C)
#undef LTL_C
        default: return cudaErrorInvalidValue;
    }
}

static size_t persist_ring_dispatch(int R) {
    switch (R) {
#define LTL_C(r) \
    case r: return persist_ring_bytes<r>();
        LTL_BATCH_RADII(LTL_C)
#undef LTL_C
        default: return 0;
    }
}

static size_t res_smem_dispatch(int R, int n) {
    switch (R) {
#define LTL_C(r) \
    case r: return res_smem_bytes<r>(n);
        LTL_BATCH_RADII(LTL_C)
#undef LTL_C
        default: return (size_t)-1;
    }
}

}  // namespace ltl

using namespace ltl;

struct BatchClass {
    Rule rule;
    PackedRule pr;
    std::vector<int> resident;   // grid ids kept in shared memory
    std::vector<int> streamed;   // grid ids streamed per step
    int* d_resident = nullptr;
    int4* d_items = nullptr;
    int n_items = 0;
    size_t res_smem = 0;
};

struct ltl_batch {
    int device = 0;
    int sms = 148;
    std::vector<BatchGrid> grids;
    std::vector<ltl_grid_desc> descs;
    std::vector<BatchClass> classes;
    std::vector<int> cls_id;
    int stream_band_rows = 64;
    long long resident_max = 0;
    BatchGrid* d_grids = nullptr;
    uint32_t* arena[2] = {nullptr, nullptr};
    size_t arena_words = 0;
    uint8_t* staging = nullptr;
    long long total_cells = 0;
    bool cur_is_a = true;
    bool no_graph = false;
    bool persistent = true;
    // persistent mode: every grid, the most work first; the CTAs' grid counter;
    // the rule classes' comparator masks
    int* d_order = nullptr;
    int n_order = 0;
    int* d_next = nullptr;
    PackedRule* d_rules = nullptr;
    BatchGroup* d_first = nullptr;     // each CTA's first task
    GridBarrier* d_barriers = nullptr; // one per grid
    unsigned int* d_err = nullptr;     // set if a group's barrier wait ran out
    int persist_ctas = 0;
    size_t persist_smem = 0;
    bool grouped = false;              // some grid has more than one CTA: cooperative launch
    bool unchecked = false;            // a grouped launch was made since d_err was last read
    bool captured = false;             // one was captured: replays come unseen, so d_err is always read
    BarrierLimit limit{};
    cudaStream_t own = nullptr, stream = nullptr, aux = nullptr;
    cudaEvent_t fork = nullptr, join = nullptr;
    // graph cache: (steps, parity) -> exec
    std::map<std::pair<int, int>, cudaGraphExec_t> graphs;
};

static void batch_release(ltl_batch* b) {
    if (!b) return;
    cudaSetDevice(b->device);
    for (auto& kv : b->graphs) cudaGraphExecDestroy(kv.second);
    for (auto& c : b->classes) {
        if (c.d_resident) cudaFree(c.d_resident);
        if (c.d_items) cudaFree(c.d_items);
    }
    if (b->d_next) cudaFree(b->d_next);
    if (b->d_order) cudaFree(b->d_order);
    if (b->d_first) cudaFree(b->d_first);
    if (b->d_barriers) cudaFree(b->d_barriers);
    if (b->d_err) cudaFree(b->d_err);
    if (b->d_rules) cudaFree(b->d_rules);
    if (b->d_grids) cudaFree(b->d_grids);
    for (auto& a : b->arena)
        if (a) cudaFree(a);
    if (b->staging) cudaFree(b->staging);
    if (b->fork) cudaEventDestroy(b->fork);
    if (b->join) cudaEventDestroy(b->join);
    if (b->aux) cudaStreamDestroy(b->aux);
    if (b->own) cudaStreamDestroy(b->own);
    delete b;
}

#define BATCH_CUDA(call)                                                                           \
    do {                                                                                           \
        cudaError_t e_ = (call);                                                                   \
        if (e_ != cudaSuccess) {                                                                   \
            cudaGetLastError(); /* reported here, not by the next launch */                        \
            ltl_set_error("%s failed: %s", #call, cudaGetErrorString(e_));                         \
            return e_ == cudaErrorMemoryAllocation ? LTL_ENOMEM : LTL_ECUDA;                       \
        }                                                                                          \
    } while (0)

static uint32_t* cur_arena(ltl_batch* b);

// A device copy of a table (allocated here).  Tables, and the words that a launch expects
// to be zero, are written in the batch's own stream: that one waits for no other, so a
// legacy-stream copy or memset could still be outstanding at the first launch.
template <class T>
static int to_device(ltl_batch* b, T** dst, const std::vector<T>& src) {
    BATCH_CUDA(cudaMalloc(dst, sizeof(T) * src.size()));
    BATCH_CUDA(cudaMemcpyAsync(*dst, src.data(), sizeof(T) * src.size(), cudaMemcpyHostToDevice, b->stream));
    return LTL_OK;
}

// Work plan: which grids are resident, and the streamed work lists.  Rebuilt
// when a shape parameter changes (the arenas' layout does not depend on it).
static int batch_plan(ltl_batch* b) {
    for (auto& kv : b->graphs) cudaGraphExecDestroy(kv.second);
    b->graphs.clear();
    for (auto& c : b->classes) {
        if (c.d_resident) cudaFree(c.d_resident);
        if (c.d_items) cudaFree(c.d_items);
        c.d_resident = nullptr;
        c.d_items = nullptr;
        c.resident.clear();
        c.streamed.clear();
        c.n_items = 0;
        c.res_smem = 0;
    }
    if (b->d_order) cudaFree(b->d_order);
    if (b->d_first) cudaFree(b->d_first);
    b->d_order = nullptr;
    b->d_first = nullptr;
    b->n_order = 0;
    b->grouped = false;
    const int count = (int)b->grids.size();
    if (b->persistent) {
        size_t smem = 0;
        for (const BatchGrid& g : b->grids) smem = std::max(smem, persist_ring_dispatch(g.R));
        // the limit of the kernel, not of this batch: another one's launches need theirs
        size_t most = 0;
        for (int r = 1; r <= kBatchMaxRadius; ++r) most = std::max(most, persist_ring_dispatch(r));
        BATCH_CUDA(cudaFuncSetAttribute(k_batch_persist, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most));
        int per_sm = 0;
        BATCH_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_batch_persist, kPersistThreads, smem));
        per_sm = std::max(per_sm, 1);
        const int ctas = b->sms * per_sm;
        std::vector<BatchCost> cost;
        for (const BatchGrid& g : b->grids) cost.emplace_back(g.n, g.nw, g.R, per_sm);
        std::vector<int> sizes;
        batch_split(cost, ctas, sizes);
        std::vector<BatchGroup> first;
        std::vector<int> order;
        for (int i = 0; i < count; ++i) {
            if (sizes[i] <= 1) order.push_back(i);
            else
                for (int r = 0; r < sizes[i]; ++r) first.push_back(BatchGroup{i, r, sizes[i]});
        }
        std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return cost[x].time(1) > cost[y].time(1); });
        b->grouped = !first.empty();
        b->persist_smem = smem;
        b->persist_ctas = (int)std::min<size_t>(ctas, first.size() + order.size());
        first.resize(b->persist_ctas, BatchGroup{0, 0, 0});
        b->n_order = (int)order.size();
        order.resize(count);  // (never empty)
        if (int r = to_device(b, &b->d_order, order)) return r;
        if (int r = to_device(b, &b->d_first, first)) return r;
        BATCH_CUDA(cudaMemsetAsync(b->d_barriers, 0, sizeof(GridBarrier) * count, b->stream));
        BATCH_CUDA(cudaStreamSynchronize(b->stream));
        return LTL_OK;
    }
    for (int i = 0; i < count; ++i) {
        BatchClass& c = b->classes[b->cls_id[i]];
        const size_t need = res_smem_dispatch(b->grids[i].R, b->grids[i].n);
        if (need <= (size_t)b->resident_max) {
            c.resident.push_back(i);
            c.res_smem = std::max(c.res_smem, need);
        } else {
            c.streamed.push_back(i);
        }
    }
    for (auto& c : b->classes)
        if (!c.resident.empty()) BATCH_CUDA(batch_prepare_dispatch(c.rule.radius));
    for (auto& c : b->classes)
        if (!c.streamed.empty()) BATCH_CUDA(batch_step_prepare_dispatch(c.rule.radius));
    for (auto& c : b->classes) {
        if (!c.resident.empty()) {
            if (int r = to_device(b, &c.d_resident, c.resident)) return r;
        }
        std::vector<int4> items;
        for (int gi : c.streamed) {
            const BatchGrid& g = b->grids[gi];
            const int strips = (g.nw + 31) / 32;
            const int band_rows = b->stream_band_rows;
            for (int r0 = 0; r0 < g.n; r0 += band_rows)
                for (int ws = 0; ws < strips; ++ws) items.push_back(make_int4(gi, r0, std::min(g.n, r0 + band_rows), ws));
        }
        c.n_items = (int)items.size();
        if (!items.empty()) {
            if (int r = to_device(b, &c.d_items, items)) return r;
        }
    }
    BATCH_CUDA(cudaStreamSynchronize(b->stream));
    return LTL_OK;
}

static int batch_build(ltl_batch* b, int flags) {
    const int count = (int)b->descs.size();
    // rule classes
    std::map<std::vector<int>, int> cls_of;
    size_t words = 0;
    long long cells = 0;
    b->grids.resize(count);
    b->cls_id.resize(count);
    int rmax = 1;
    for (int i = 0; i < count; ++i) {
        const ltl_grid_desc& d = b->descs[i];
        std::vector<int> key = {d.radius, d.smin, d.smax, d.bmin, d.bmax};
        auto it = cls_of.find(key);
        if (it == cls_of.end()) {
            BatchClass c;
            c.rule = Rule{d.radius, d.smin, d.smax, d.bmin, d.bmax};
            c.pr = make_packed_rule(c.rule);
            it = cls_of.emplace(key, (int)b->classes.size()).first;
            b->classes.push_back(c);
        }
        b->cls_id[i] = it->second;
        BatchGrid g{};
        g.n = d.n;
        g.nw = (d.n + 31) / 32;
        g.wp = (g.nw + 3) / 4 * 4;
        g.R = d.radius;
        g.off = (long long)words;
        g.cell_off = cells;
        words += (size_t)g.n * g.wp;
        words = (words + 31) / 32 * 32;
        cells += (long long)g.n * g.n;
        g.cls = it->second;
        b->grids[i] = g;
        rmax = std::max(rmax, d.radius);
    }
    b->arena_words = words + 64;
    b->total_cells = cells;
    b->stream_band_rows = (int)tuning_lookup("batch", -1, 0, "stream_band_rows", 64);
    b->resident_max = (flags & LTL_BATCH_STREAM_ALL) ? 0
                                                     : tuning_lookup("batch", -1, 0, "resident_max_bytes", kResSmemLimit);
    b->persistent = !(flags & LTL_BATCH_STREAM_ALL) && tuning_lookup("batch", -1, 0, "persistent", 1) != 0;
    BATCH_CUDA(cudaMalloc(&b->d_next, sizeof(int)));
    BATCH_CUDA(cudaMalloc(&b->d_err, sizeof(unsigned int)));
    BATCH_CUDA(cudaMemsetAsync(b->d_err, 0, sizeof(unsigned int), b->stream));
    BATCH_CUDA(cudaMalloc(&b->d_barriers, sizeof(GridBarrier) * count));
    {
        std::vector<PackedRule> rules;
        for (auto& c : b->classes) rules.push_back(c.pr);
        if (int r = to_device(b, &b->d_rules, rules)) return r;
    }
    if (int r = to_device(b, &b->d_grids, b->grids)) return r;
    for (auto& a : b->arena) {
        BATCH_CUDA(cudaMalloc(&a, b->arena_words * sizeof(uint32_t)));
        BATCH_CUDA(cudaMemsetAsync(a, 0, b->arena_words * sizeof(uint32_t), b->stream));
    }
    BATCH_CUDA(cudaMalloc(&b->staging, (size_t)std::max<long long>(cells, 1)));
    return batch_plan(b);
}

extern "C" int ltl_batch_set_param(ltl_batch* b, const char* name, long long value) {
    if (!b || !name) {
        ltl_set_error("ltl_batch_set_param: bad arguments");
        return LTL_EINVAL;
    }
    BATCH_CUDA(cudaSetDevice(b->device));
    BATCH_CUDA(cudaStreamSynchronize(b->stream));
    if (std::strcmp(name, "stream_band_rows") == 0) {
        if (value < 8 || value > 4096) {
            ltl_set_error("ltl_batch_set_param: stream_band_rows must be in [8, 4096]");
            return LTL_EINVAL;
        }
        b->stream_band_rows = (int)value;
    } else if (std::strcmp(name, "persistent") == 0) {
        if (value != 0 && value != 1) {
            ltl_set_error("ltl_batch_set_param: persistent must be 0 or 1");
            return LTL_EINVAL;
        }
        b->persistent = value != 0;
    } else if (std::strcmp(name, "resident_max_bytes") == 0) {
        if (value < 0 || value > kResSmemLimit) {
            ltl_set_error("ltl_batch_set_param: resident_max_bytes must be in [0, %d]", kResSmemLimit);
            return LTL_EINVAL;
        }
        b->resident_max = value;
    } else if (std::strcmp(name, "inject_missing_arrival") == 0) {
        if (value != 0 && (value < 1000000 || value > 10000000000ll)) {
            ltl_set_error("ltl_batch_set_param: inject_missing_arrival must be 0 or a wait limit in [1e6, 1e10] ns");
            return LTL_EINVAL;
        }
        b->limit = BarrierLimit{};
        if (value) b->limit = BarrierLimit{(unsigned long long)value, 1u};
    } else {
        ltl_set_error("ltl_batch_set_param: unknown parameter '%s'", name);
        return LTL_EINVAL;
    }
    return batch_plan(b);
}

extern "C" int ltl_batch_create(ltl_batch** out, int device, const ltl_grid_desc* descs, int count, int flags) {
    if (!out || !descs || count < 1) {
        ltl_set_error("ltl_batch_create: bad arguments");
        return LTL_EINVAL;
    }
    *out = nullptr;
    for (int i = 0; i < count; ++i) {
        const ltl_grid_desc& d = descs[i];
        if (d.n < 1 || d.radius < 1 || d.n < d.radius) {
            ltl_set_error("ltl_batch_create: grid %d: need n >= radius >= 1 (n=%d, radius=%d)", i, d.n, d.radius);
            return LTL_EINVAL;
        }
        if (d.radius > kBatchMaxRadius) {
            ltl_set_error("ltl_batch_create: grid %d: batched grids support radius <= 16 (got %d)", i, d.radius);
            return LTL_EUNSUPPORTED;
        }
    }
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev) {
        ltl_set_error("ltl_batch_create: CUDA device %d not available", device);
        return LTL_ECUDA;
    }
    ltl_batch* b = new (std::nothrow) ltl_batch();
    if (!b) return LTL_ENOMEM;
    b->device = device;
    b->descs.assign(descs, descs + count);
    cudaSetDevice(device);
    cudaDeviceGetAttribute(&b->sms, cudaDevAttrMultiProcessorCount, device);
    cudaError_t se = cudaStreamCreateWithFlags(&b->own, cudaStreamNonBlocking);
    if (se == cudaSuccess) se = cudaStreamCreateWithFlags(&b->aux, cudaStreamNonBlocking);
    if (se == cudaSuccess) se = cudaEventCreateWithFlags(&b->fork, cudaEventDisableTiming);
    if (se == cudaSuccess) se = cudaEventCreateWithFlags(&b->join, cudaEventDisableTiming);
    if (se != cudaSuccess) {
        ltl_set_error("ltl_batch_create: stream/event creation failed: %s", cudaGetErrorString(se));
        batch_release(b);
        return LTL_ECUDA;
    }
    b->stream = b->own;
    b->no_graph = (flags & LTL_BATCH_NO_GRAPH) != 0;
    int rc = batch_build(b, flags);
    if (rc != LTL_OK) {
        batch_release(b);
        return rc;
    }
    *out = b;
    return LTL_OK;
}

extern "C" int ltl_batch_destroy(ltl_batch* b) {
    if (!b) return LTL_OK;
    cudaSetDevice(b->device);
    cudaStreamSynchronize(b->stream);
    batch_release(b);
    return LTL_OK;
}

extern "C" int ltl_batch_set_stream(ltl_batch* b, void* stream) {
    if (!b) {
        ltl_set_error("null batch");
        return LTL_EINVAL;
    }
    cudaStream_t s = stream ? (cudaStream_t)stream : b->own;
    if (s != b->stream) {
        for (auto& kv : b->graphs) cudaGraphExecDestroy(kv.second);
        b->graphs.clear();
    }
    b->stream = s;
    return LTL_OK;
}

static uint32_t* cur_arena(ltl_batch* b) { return b->arena[b->cur_is_a ? 0 : 1]; }
static uint32_t* nxt_arena(ltl_batch* b) { return b->arena[b->cur_is_a ? 1 : 0]; }

// Waits for the stream; did a group's barrier wait run out since this was last asked?
static int wait_groups(ltl_batch* b) {
    unsigned int flag = 0;
    if (b->unchecked || b->captured)
        BATCH_CUDA(cudaMemcpyAsync(&flag, b->d_err, sizeof(flag), cudaMemcpyDeviceToHost, b->stream));
    BATCH_CUDA(cudaStreamSynchronize(b->stream));
    b->unchecked = false;
    if (!flag) return LTL_OK;
    BATCH_CUDA(cudaMemsetAsync(b->d_err, 0, sizeof(flag), b->stream));
    BATCH_CUDA(cudaMemsetAsync(b->d_barriers, 0, sizeof(GridBarrier) * b->grids.size(), b->stream));
    BATCH_CUDA(cudaStreamSynchronize(b->stream));
    ltl_set_error("batch kernel reported a bounded-wait timeout; the grids are unspecified until the next upload");
    return LTL_ETIMEOUT;
}

extern "C" int ltl_batch_upload_all(ltl_batch* b, const uint8_t* cells) {
    if (!b || !cells) {
        ltl_set_error("ltl_batch_upload_all: bad arguments");
        return LTL_EINVAL;
    }
    BATCH_CUDA(cudaSetDevice(b->device));
    BATCH_CUDA(cudaMemcpyAsync(b->staging, cells, (size_t)b->total_cells, cudaMemcpyHostToDevice, b->stream));
    const int count = (int)b->grids.size();
    for (int first = 0; first < count; first += 65535) {
        dim3 g(16, (unsigned)std::min(65535, count - first));
        k_batch_pack<<<g, 256, 0, b->stream>>>(b->staging, cur_arena(b), b->d_grids, first, b->d_barriers);
    }
    BATCH_CUDA(cudaGetLastError());
    BATCH_CUDA(cudaStreamSynchronize(b->stream));
    return LTL_OK;
}

extern "C" int ltl_batch_download_all(ltl_batch* b, uint8_t* cells) {
    if (!b || !cells) {
        ltl_set_error("ltl_batch_download_all: bad arguments");
        return LTL_EINVAL;
    }
    BATCH_CUDA(cudaSetDevice(b->device));
    const int count = (int)b->grids.size();
    for (int first = 0; first < count; first += 65535) {
        dim3 g(16, (unsigned)std::min(65535, count - first));
        k_batch_unpack<<<g, 256, 0, b->stream>>>(cur_arena(b), b->staging, b->d_grids, first);
    }
    BATCH_CUDA(cudaGetLastError());
    BATCH_CUDA(cudaMemcpyAsync(cells, b->staging, (size_t)b->total_cells, cudaMemcpyDeviceToHost, b->stream));
    return wait_groups(b);
}

extern "C" int ltl_batch_upload(ltl_batch* b, int grid, const uint8_t* inner, size_t pitch) {
    if (!b || !inner || grid < 0 || grid >= (int)b->grids.size() || pitch < (size_t)b->grids[grid].n) {
        ltl_set_error("ltl_batch_upload: bad arguments");
        return LTL_EINVAL;
    }
    BATCH_CUDA(cudaSetDevice(b->device));
    const BatchGrid& g = b->grids[grid];
    BATCH_CUDA(cudaMemcpy2DAsync(b->staging + g.cell_off, g.n, inner, pitch, g.n, g.n, cudaMemcpyHostToDevice,
                                 b->stream));
    k_batch_pack<<<dim3(16, 1), 256, 0, b->stream>>>(b->staging, cur_arena(b), b->d_grids, grid, b->d_barriers);
    BATCH_CUDA(cudaGetLastError());
    BATCH_CUDA(cudaStreamSynchronize(b->stream));
    return LTL_OK;
}

extern "C" int ltl_batch_download(ltl_batch* b, int grid, uint8_t* inner, size_t pitch) {
    if (!b || !inner || grid < 0 || grid >= (int)b->grids.size() || pitch < (size_t)b->grids[grid].n) {
        ltl_set_error("ltl_batch_download: bad arguments");
        return LTL_EINVAL;
    }
    BATCH_CUDA(cudaSetDevice(b->device));
    const BatchGrid& g = b->grids[grid];
    k_batch_unpack<<<dim3(16, 1), 256, 0, b->stream>>>(cur_arena(b), b->staging, b->d_grids, grid);
    BATCH_CUDA(cudaGetLastError());
    BATCH_CUDA(cudaMemcpy2DAsync(inner, pitch, b->staging + g.cell_off, g.n, g.n, g.n, cudaMemcpyDeviceToHost,
                                 b->stream));
    return wait_groups(b);
}

// Enqueue `steps` generations of every grid (stream-ordered on b->stream).
// On failure, `what` names the call that failed.
static cudaError_t enqueue_steps(ltl_batch* b, int steps, const char** what) {
    cudaError_t e = cudaSuccess;
    uint32_t* a0 = cur_arena(b);
    uint32_t* a1 = nxt_arena(b);
    if (b->persistent) {
        *what = "grid counter reset";
        e = cudaMemsetAsync(b->d_next, 0, sizeof(int), b->stream);
        if (e == cudaSuccess) {
            *what = "persistent kernel launch";
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = dim3(b->persist_ctas);
            cfg.blockDim = dim3(kPersistThreads);
            cfg.dynamicSmemBytes = b->persist_smem;
            cfg.stream = b->stream;
            cudaLaunchAttribute at{};
            at.id = cudaLaunchAttributeCooperative;
            at.val.cooperative = b->grouped;
            cfg.attrs = &at;
            cfg.numAttrs = 1;
            e = cudaLaunchKernelEx(&cfg, k_batch_persist, a0, a1, (const BatchGrid*)b->d_grids,
                                   (const PackedRule*)b->d_rules, (const BatchGroup*)b->d_first,
                                   BatchWaits{b->d_barriers, b->d_err, b->limit}, (const int*)b->d_order, b->n_order,
                                   b->d_next, steps);
        }
        return e;
    }
    bool any_res = false;
    for (auto& c : b->classes) any_res |= !c.resident.empty();
    if (any_res) {
        *what = "fork event record";
        e = cudaEventRecord(b->fork, b->stream);
        if (e == cudaSuccess) {
            *what = "fork stream wait";
            e = cudaStreamWaitEvent(b->aux, b->fork, 0);
        }
        uint32_t* dst = (steps % 2) ? a1 : a0;
        for (auto& c : b->classes) {
            if (c.resident.empty() || e != cudaSuccess) continue;
            *what = "resident kernel launch";
            e = batch_resident_dispatch(c.rule.radius, a0, dst, b->d_grids, c.d_resident, (int)c.resident.size(),
                                        steps, c.pr, c.res_smem, b->sms, b->aux);
        }
        if (e == cudaSuccess) {
            *what = "join event record";
            e = cudaEventRecord(b->join, b->aux);
        }
    }
    for (int s = 0; s < steps && e == cudaSuccess; ++s) {
        const uint32_t* src = (s % 2) ? a1 : a0;
        uint32_t* dst = (s % 2) ? a0 : a1;
        for (auto& c : b->classes) {
            if (c.n_items == 0 || e != cudaSuccess) continue;
            *what = "streamed step kernel launch";
            e = batch_step_dispatch(c.rule.radius, src, dst, b->d_grids, c.d_items, c.n_items, c.pr, b->sms,
                                    b->stream);
        }
    }
    if (any_res && e == cudaSuccess) {
        *what = "join stream wait";
        e = cudaStreamWaitEvent(b->stream, b->join, 0);
    }
    return e;
}

extern "C" int ltl_batch_step(ltl_batch* b, int steps) {
    if (!b || steps < 0) {
        ltl_set_error("ltl_batch_step: bad arguments");
        return LTL_EINVAL;
    }
    if (steps == 0) return LTL_OK;
    BATCH_CUDA(cudaSetDevice(b->device));
    if (b->persistent && b->grouped) {
        cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
        if (b->no_graph) BATCH_CUDA(cudaStreamIsCapturing(b->stream, &capture));
        b->unchecked = true;
        b->captured = b->captured || capture != cudaStreamCaptureStatusNone;
    }
    const char* what = "";
    if (b->no_graph) {
        cudaError_t e = enqueue_steps(b, steps, &what);
        if (e != cudaSuccess) {
            cudaGetLastError();
            ltl_set_error("ltl_batch_step: %s failed: %s", what, cudaGetErrorString(e));
            return LTL_ECUDA;
        }
        if (steps % 2) b->cur_is_a = !b->cur_is_a;
        return LTL_OK;
    }
    const std::pair<int, int> key(steps, b->cur_is_a ? 0 : 1);
    auto it = b->graphs.find(key);
    if (it == b->graphs.end()) {
        cudaGraph_t g = nullptr;
        BATCH_CUDA(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
        cudaError_t e = enqueue_steps(b, steps, &what);
        cudaError_t e2 = cudaStreamEndCapture(b->stream, &g);
        if (e != cudaSuccess || e2 != cudaSuccess) {
            if (g) cudaGraphDestroy(g);
            ltl_set_error("ltl_batch_step: graph capture failed at %s: %s / end capture: %s", what,
                          cudaGetErrorString(e), cudaGetErrorString(e2));
            cudaGetLastError();
            return LTL_ECUDA;
        }
        cudaGraphExec_t ex = nullptr;
        cudaError_t e3 = cudaGraphInstantiate(&ex, g, 0);
        cudaGraphDestroy(g);
        if (e3 != cudaSuccess) {
            cudaGetLastError();
            ltl_set_error("ltl_batch_step: graph instantiate failed: %s", cudaGetErrorString(e3));
            return LTL_ECUDA;
        }
        it = b->graphs.emplace(key, ex).first;
    }
    BATCH_CUDA(cudaGraphLaunch(it->second, b->stream));
    if (steps % 2) b->cur_is_a = !b->cur_is_a;
    return LTL_OK;
}

extern "C" int ltl_batch_synchronize(ltl_batch* b) {
    if (!b) {
        ltl_set_error("null batch");
        return LTL_EINVAL;
    }
    BATCH_CUDA(cudaSetDevice(b->device));
    return wait_groups(b);
}

extern "C" int ltl_batch_info(const ltl_batch* b, long long* cells, long long* device_bytes, int* temporal_depth) {
    if (!b) {
        ltl_set_error("null batch");
        return LTL_EINVAL;
    }
    if (cells) *cells = b->total_cells;
    if (device_bytes) *device_bytes = (long long)(2 * b->arena_words * 4 + b->total_cells);
    if (temporal_depth) {
        // grids that run every generation of an ltl_batch_step inside one launch
        int res = 0;
        if (b->persistent) res = (int)b->grids.size();
        else
            for (auto& c : b->classes) res += (int)c.resident.size();
        *temporal_depth = res;
    }
    return LTL_OK;
}
