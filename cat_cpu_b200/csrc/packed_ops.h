// packed_ops.h -- what k_packed_radius.cu defines for each radius.
//
// A part per radius, so that each is a CUDA module of its own: the first use of any kernel
// loads its whole module, and a program uses a radius or two.  With all 32 radii in one
// module the first packed (or default) solver of a process took 22 ms to create; a part
// takes 0.8 ms.
#pragma once

#include "ltl_kernels.h"

namespace ltl {

struct PackedRule;  // packed_core.cuh

template <int R>
struct PackedOps {
    static cudaError_t prepare(const PackedFrame& f, bool walk, int sms);
    static cudaError_t step(const PackedFrame& cur, const PackedFrame& nxt, const PackedRule& pr, int band_rows,
                            cudaStream_t s);
    static bool runs(const PackedFrame& f, int sms);
    static cudaError_t run(const PackedFrame& cur, const PackedFrame& nxt, const PackedRule& pr, int steps, int sms,
                           const PackedRun& run, cudaStream_t s);
};

}  // namespace ltl
