// k_packed.cu -- K3: bit-packed LtL step, by radius (kernels: k_packed_radius.cu).
#include "packed_core.cuh"
#include "packed_ops.h"

namespace ltl {

bool packed_supported(int n, int radius) { return radius >= 1 && radius <= 32 && n >= radius; }

static int device_sms() {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

cudaError_t packed_prepare(const PackedFrame& f, int radius, bool walk) {
    const int sms = device_sms();
    switch (radius) {
#define LTL_PP(r) \
    case r: return PackedOps<r>::prepare(f, walk, sms);
        LTL_PACKED_RADII(LTL_PP)
#undef LTL_PP
        default: return cudaSuccess;
    }
}

cudaError_t launch_packed_step(const PackedFrame& cur, const PackedFrame& nxt, const Rule& rule, int band_rows,
                               cudaStream_t s) {
    const PackedRule pr = make_packed_rule(rule);
    switch (rule.radius) {
#define LTL_PR(r) \
    case r: return PackedOps<r>::step(cur, nxt, pr, band_rows, s);
        LTL_PACKED_RADII(LTL_PR)
#undef LTL_PR
        default: return cudaErrorInvalidValue;
    }
}

bool packed_runs(const PackedFrame& f, int radius) {
    const int sms = device_sms();
    switch (radius) {
#define LTL_PR(r) \
    case r: return PackedOps<r>::runs(f, sms);
        LTL_PACKED_RADII(LTL_PR)
#undef LTL_PR
        default: return false;
    }
}

cudaError_t launch_packed_run(const PackedFrame& cur, const PackedFrame& nxt, const Rule& rule, int steps,
                              const PackedRun& run, cudaStream_t s) {
    const PackedRule pr = make_packed_rule(rule);
    const int sms = device_sms();
    switch (rule.radius) {
#define LTL_PR(r) \
    case r: return PackedOps<r>::run(cur, nxt, pr, steps, sms, run, s);
        LTL_PACKED_RADII(LTL_PR)
#undef LTL_PR
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace ltl
