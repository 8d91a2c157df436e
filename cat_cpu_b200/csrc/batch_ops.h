// batch_ops.h -- a batch's grids, and what k_batch_radius.cu defines for each radius: the
// launches of per-generation mode.  A part (a CUDA module) per radius, as in packed_ops.h:
// batches that run persistently load none of them.
#pragma once

#include "ltl_kernels.h"

namespace ltl {

struct PackedRule;  // packed_core.cuh

struct BatchGrid {
    long long off;       // word offset of the grid's packed frame in an arena
    long long cell_off;  // byte offset of the grid in the dense staging buffer
    int n, nw, wp;       // cells per side, words per row, row pitch in words (a multiple of 4)
    int R;
    int cls;             // rule class
};

constexpr int kBatchWarps = 4;
constexpr int kResThreads = 1024;
constexpr int kResSmemLimit = 220 * 1024;
constexpr int kBatchMaxRadius = 16;

template <int R>
struct BatchOps {
    // one generation of the streamed grids of a rule class: items are (grid, r0, r1, word strip)
    static cudaError_t step(const uint32_t* cur, uint32_t* nxt, const BatchGrid* grids, const int4* items, int n_items,
                            const PackedRule& pr, int sms, cudaStream_t s);
    // `steps` generations of the resident ones
    static cudaError_t resident(const uint32_t* src, uint32_t* dst, const BatchGrid* grids, const int* list, int n_list,
                                int steps, const PackedRule& pr, size_t smem, int sms, cudaStream_t s);
    // attributes, outside any stream capture
    static cudaError_t prepare_step();
    static cudaError_t prepare_resident();
};

}  // namespace ltl
