// Host-side plans of the launches whose CTAs wait for one another, compiled as they are
// (test_run_plans.py): the batch's groups (batch_split.h) and the small packed grids'
// blocks of generations (packed_tile.cuh).
#include <cstdint>

#include <cuda_runtime.h>

static inline uint32_t __funnelshift_r(uint32_t, uint32_t, uint32_t) { return 0; }
static inline uint32_t __funnelshift_rc(uint32_t, uint32_t, uint32_t) { return 0; }
static inline uint32_t __funnelshift_l(uint32_t, uint32_t, uint32_t) { return 0; }
template <class T>
static T __ldg(const T* p) { return *p; }

#include "batch_split.h"
#include "packed_tile.cuh"

using namespace ltl;

// CTAs per grid into sizes, and the model's time of a generation for each.
extern "C" void batch_split_host(const int* n, const int* radius, int count, int ctas, int per_sm, int* sizes,
                                 double* times, double* alone) {
    std::vector<BatchCost> cost;
    for (int i = 0; i < count; ++i) cost.emplace_back(n[i], (n[i] + 31) / 32, radius[i], per_sm);
    std::vector<int> got;
    batch_split(cost, ctas, got);
    for (int i = 0; i < count; ++i) {
        sizes[i] = got[i];
        times[i] = cost[i].time(got[i]);
        alone[i] = cost[i].time(1);
    }
}

// Generations of each block into gens; returns the number of blocks.
extern "C" int run_blocks_host(int steps, int depth, int* gens) {
    int blocks = run_blocks(steps, depth), k = 0;
    const int all = blocks;
    for (int s = 0; s < steps; --blocks) s += gens[k++] = block_generations(steps - s, blocks);
    return k == all ? k : -1;
}
