// k_tensor_set.cu -- the tensor step's kernels (tensor_step.cuh) of one rule-lane mode and
// number of K steps: LTL_TENSOR_MODE, LTL_TENSOR_NG (build.py compiles a part for each).
//
// Parts, so that each is a CUDA module of its own: the first use of any kernel loads its
// whole module, and a program uses one or two of these sets.  In one module the first
// tensor solver of a process took 15.6 ms to create.
#include "tensor_step.cuh"

namespace ltl {

template <int MODE, int NG, bool RUN>
static TcKernel pick_form(int form) {
    constexpr bool XT = tensor_xt(MODE, true, NG);
    switch (form) {
        case kFast: return k_tensor_step<MODE, kFast, NG, XT, RUN>;
        case kFastSeam: return k_tensor_step<MODE, kFastSeam, NG, XT, RUN>;
        default: return k_tensor_step<MODE, kGather, NG, false, RUN>;
    }
}

template <int MODE, int NG>
TcKernel tensor_kernel(int form, bool run) {
    return run ? pick_form<MODE, NG, true>(form) : pick_form<MODE, NG, false>(form);
}

#ifdef LTL_TENSOR_MODE
template TcKernel tensor_kernel<LTL_TENSOR_MODE, LTL_TENSOR_NG>(int form, bool run);
#else
#define LTL_ALL(mode, ng) template TcKernel tensor_kernel<mode, ng>(int form, bool run);
LTL_TENSOR_SETS(LTL_ALL)
#undef LTL_ALL
#endif

}  // namespace ltl
