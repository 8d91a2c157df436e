// k_tensor.cu -- K2, host side: the tensor step's tile geometry, plans and launches
// (kernel: tensor_step.cuh).
#include <algorithm>
#include <cstdio>
#include <cstring>

#include "tensor_step.cuh"

namespace ltl {

// More than half of an SM's 228 KB: a CTA takes all of the SM's tensor memory, and two
// launches of many generations that shared SMs could each hold it where the other waits
// for it.  (The registers keep CTAs apart as well, but that is the compiler's choice.)
constexpr int kSmemFloor = 116 * 1024;

struct TensorPlan {
    TcParams prm[2];  // source frame a -> b, b -> a
    TcKernel kernel, run;  // one generation, many
    bool runs;             // small enough for many per launch
    int smem_bytes;
    int grid;
    int operand_bits;  // product-2 operand: 8 (u8) or 16 (f16)
    unsigned int* err;
    GridBarrier* barrier;  // zero whenever no launch that failed has used it
};

static TcKernel pick_kernel(int mode, int ng, int form, bool run) {
#define LTL_PICK(m, k) \
    if (mode == m && ng == k) return tensor_kernel<m, k>(form, run);
    LTL_TENSOR_SETS(LTL_PICK)
#undef LTL_PICK
    return nullptr;
}

// Largest radius of the tensor step.  Row sums 2R+1 <= 255 travel as u8; R = 128
// (row sums up to 257) as f16.  Above it the X tiles of three or more row blocks
// and the f16 operands no longer fit one SM's shared memory twice over.
constexpr int kTensorMaxRadius = 128;

bool tensor_supported(int n, int radius, char* why, size_t why_len) {
    if (radius < 1 || radius > kTensorMaxRadius) {
        snprintf(why, why_len, "tensor variant supports 1 <= R <= %d (got %d)", kTensorMaxRadius, radius);
        return false;
    }
    if (n < radius) {
        snprintf(why, why_len, "n < R");
        return false;
    }
    return true;
}

// Lane constants of the interval rule on the box count B (centre included):
// a live cell survives iff smin+1 <= B <= smax+1, a dead one is born iff
// bmin <= B <= bmax.  For a lane of `bits` bits whose top bit is the marker,
// nlo = top - lo (B + nlo has the marker set iff B >= lo) and hiH = top + hi
// (hiH - B has it set iff B <= hi); empty intervals become lo = top, hi = 0.
static void lane_consts(int lo, int hi, int bits, int& nlo, int& hiH) {
    const int top = 1 << (bits - 1);
    if (lo < 0) lo = 0;
    if (hi > top - 1) hi = top - 1;
    if (hi < lo || lo > top - 1) {
        lo = top;
        hi = 0;
    }
    nlo = top - lo;
    hiH = top + hi;
}

// The same for one 32-bit lane (marker bit 31).  The lane holds either the
// box count B itself (s32) or, with `fbits`, the bit pattern of the f32 value
// B + off; both are below 2^31 and ordered like B, so the thresholds are
// transformed the same way.  An empty interval gives nlo = 0 (B + 0 never has
// bit 31 set).
static void lane_consts32(int lo, int hi, int maxB, bool fbits, int off, uint32_t& nlo, uint32_t& hiH) {
    if (lo < 0) lo = 0;
    if (hi > maxB) hi = maxB;
    if (hi < lo) {
        nlo = 0u;
        hiH = 0x80000000u;
        return;
    }
    uint32_t l = (uint32_t)lo, h = (uint32_t)hi;
    if (fbits) {
        const float fl = (float)(lo + off), fh = (float)(hi + off);
        memcpy(&l, &fl, 4);
        memcpy(&h, &fh, 4);
    }
    nlo = 0x80000000u - l;
    hiH = 0x80000000u + h;
}

// Tile geometry for radius R (also restated in tests/test_tensor_tiles.py):
//   Tc = 128 output columns per tile (H and C, two buffers each, fill the 512
//          TMEM columns);
//   PADC = 16 + 32a >= R columns of halo on each side of the output columns
//          (16 mod 32, so that every X group straddles two packed words by halves);
//   nb = 1 row block for R <= 32 (Tr = 128 - 2R output rows per tile), else
//          enough 128-row blocks for Tr = 128 rows plus 2R halo rows;
//   ng = ceil((PADC + Tc + R) / 32) product-1 K steps reach every X column
//          that any output column of the tile needs;
//   mode = the rule lanes and product-2 operand (TcMode);
//   fast = the packed words of the next units staged through shared memory,
//          where n allows it and the ring fits beside the deepest X ring.
struct TensorGeometry {
    int PADC, Tr, nb, ng, mode, stages;
    bool fast;
};

static int tensor_mode(int R) {
    if ((2 * R + 1) * (2 * R + 1) <= 127) return kLanes8;
    if ((2 * R + 1) * (2 * R + 1) < (1 << 15)) return kLanes16;
    return 2 * R + 1 <= 255 ? kLanes32 : kF16;
}

static bool tensor_geometry(int R, bool fast_ok, TensorGeometry& G) {
    G.PADC = R <= 16 ? 16 : 16 + 32 * ((R - 16 + 31) / 32);
    G.nb = R <= 32 ? 1 : (128 + 2 * R + 127) / 128;
    G.Tr = G.nb == 1 ? 128 - 2 * R : std::min(128, 128 * G.nb - 2 * R);
    G.ng = (G.PADC + kTc + R + 31) / 32;
    G.mode = tensor_mode(R);
    if (G.Tr < 1 || R > kTensorMaxRadius || 2 * R + 1 + kF16Offset > 2048) return false;
    if (tensor_xt(G.mode, fast_ok, G.ng)) {
        // X in tensor memory: kXtStages stages of TMEM columns, no X in shared memory
        G.stages = kXtStages;
        G.fast = true;
        return smem_layout(G.stages, G.ng, G.nb, true, G.mode, true).total + 1024 <= kSmemLimit;
    }
    // the deepest X ring that fits, with the word ring where possible
    for (int f = fast_ok ? 1 : 0; f >= 0; --f) {
        for (int st = kMaxStages; st >= 2; --st) {
            if (smem_layout(st, G.ng, G.nb, f != 0, G.mode).total + 1024 <= kSmemLimit) {
                G.stages = st;
                G.fast = f != 0;
                return true;
            }
        }
    }
    return false;
}

TensorPlan* tensor_plan_create(const PackedFrame& a, const PackedFrame& b, const Rule& rule, int device,
                               GridBarrier* barrier, unsigned int* err, char* why, size_t why_len) {
    if (!tensor_supported(a.n, rule.radius, why, why_len)) return nullptr;
    int major = 0;
    cudaDeviceGetAttribute(&major, cudaDevAttrComputeCapabilityMajor, device);
    if (major != 10) {
        snprintf(why, why_len, "tcgen05 needs an sm_100 device (compute capability %d.x)", major);
        return nullptr;
    }
    if (a.HW < 1 || b.HW < 1) {
        snprintf(why, why_len, "packed frames need a halo word");
        return nullptr;
    }
    const int R = rule.radius;
    const int nw = a.nw;
    // one correction wraps a row (rows span [-R, n + 128 nb)) and a word index
    // (words span [-4, nw + ng)); groups are word halves
    const int nb_of_r = R <= 32 ? 1 : (128 + 2 * R + 127) / 128;
    // where 32 does not divide n, rows of fewer tiles than this are gathered: too many of them
    // reach over the seam (us per generation, staged / gathered: 1000^2 R = 5 5.9 / 4.8, R = 113
    // 19.6 / 12.4, 1500^2 R = 8 7.0 / 6.7, R = 90 16.2 / 12.9; 2001^2 R = 8 7.1 / 7.0, R = 16 7.9 /
    // 8.8, R = 90 19.9 / 22.3, R = 113 24.2 / 22.3; 3001^2 R = 64 20 / 28)
    constexpr int kSeamTiles = 16;
    const bool fast_ok = nw >= 4 && a.n >= 128 * nb_of_r + R && (a.n % 32 == 0 || (a.n + kTc - 1) / kTc >= kSeamTiles);
    TensorGeometry G{};
    if (!tensor_geometry(R, fast_ok, G)) {
        snprintf(why, why_len, "no tile shape for R=%d", R);
        return nullptr;
    }
    const bool fast = G.fast;
    TensorPlan* P = new TensorPlan();
    P->operand_bits = G.mode == kF16 ? 16 : 8;
    uint32_t nlo_d, hiH_d, nlo_s, hiH_s, bcast = 1u;
    if (G.mode >= kLanes32) {
        const int maxB = (2 * R + 1) * (2 * R + 1);
        const bool fb = G.mode == kF16;
        const int off = fb ? kF16Offset * (2 * R + 1) : 0;
        lane_consts32(rule.bmin, rule.bmax, maxB, fb, off, nlo_d, hiH_d);
        lane_consts32(rule.smin + 1, rule.smax + 1, maxB, fb, off, nlo_s, hiH_s);
    } else {
        const int bits = G.mode == kLanes16 ? 16 : 8;
        bcast = G.mode == kLanes16 ? 0x00010001u : 0x01010101u;
        int a0, b0, a1, b1;
        lane_consts(rule.bmin, rule.bmax, bits, a0, b0);
        lane_consts(rule.smin + 1, rule.smax + 1, bits, a1, b1);
        nlo_d = (uint32_t)a0;
        hiH_d = (uint32_t)b0;
        nlo_s = (uint32_t)a1;
        hiH_s = (uint32_t)b1;
    }
    const PackedFrame* src[2] = {&a, &b};
    const PackedFrame* dst[2] = {&b, &a};
    for (int i = 0; i < 2; ++i) {
        TcParams& q = P->prm[i];
        q.src = src[i]->words + (size_t)src[i]->HR * src[i]->wpitch + src[i]->HW;
        q.dst = dst[i]->words + (size_t)dst[i]->HR * dst[i]->wpitch + dst[i]->HW;
        q.wpitch = (long long)a.wpitch;
        q.n = a.n;
        q.nw = nw;
        q.R = R;
        q.PADC = G.PADC;
        q.Tr = G.Tr;
        q.nb = G.nb;
        q.stages = G.stages;
        q.tiles_x = (a.n + kTc - 1) / kTc;
        q.tiles_y = (a.n + G.Tr - 1) / G.Tr;
        q.nlo0 = nlo_d * bcast;
        q.dlo = nlo_s - nlo_d;
        q.hiH0 = hiH_d * bcast;
        q.dhi = hiH_s - hiH_d;
    }
    for (auto& q : P->prm) {
        q.err = err;
        q.barrier = barrier;
        q.steps = 1;
        q.wait_ns = kWaitLimitNs;
        q.inject_missing_commit = 0;
    }
    const int form = !fast ? kGather : (a.n % 32 == 0 ? kFast : kFastSeam);
    P->kernel = pick_kernel(G.mode, G.ng, form, false);
    P->run = pick_kernel(G.mode, G.ng, form, true);
    if (!P->kernel) {
        snprintf(why, why_len, "no kernel instantiation for R=%d", R);
        delete P;
        return nullptr;
    }
    P->smem_bytes = std::max(smem_layout(G.stages, G.ng, G.nb, fast, G.mode, tensor_xt(G.mode, fast, G.ng)).total + 1024,
                             kSmemFloor);
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    P->grid = std::min(P->prm[0].tiles_x * P->prm[0].tiles_y, sms);
    // units of a generation per CTA: with many, the run's longer loops cost more than
    // the launches (16384^2 R = 5 115 us per generation in launches of one, 128 in one
    // launch; 8192^2 R = 5 33.5 / 34.3; 4096^2 R = 5 12.6 / 11.5, R = 100 33.5 / 32.5)
    P->runs = (long long)P->prm[0].tiles_x * P->prm[0].tiles_y * G.nb <= 24ll * P->grid;
    // the kernel's limit, not this plan's: plans of other radii launch the same kernel with more
    cudaError_t ae = cudaFuncSetAttribute(P->kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit);
    if (ae == cudaSuccess && P->runs)
        ae = cudaFuncSetAttribute(P->run, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemLimit);
    if (ae != cudaSuccess) {
        snprintf(why, why_len, "cannot reserve %d bytes of shared memory", P->smem_bytes);
        delete P;
        return nullptr;
    }
    return P;
}

void tensor_plan_destroy(TensorPlan* p) { delete p; }

int tensor_plan_depth(const TensorPlan*) { return 1; }

void tensor_plan_set_wait(TensorPlan* p, unsigned long long ns, int inject_missing_commit) {
    for (auto& q : p->prm) {
        q.wait_ns = ns;
        q.inject_missing_commit = inject_missing_commit;
    }
}
int tensor_plan_operand_bits(const TensorPlan* p) { return p ? p->operand_bits : 0; }

bool tensor_plan_runs(const TensorPlan* p) { return p->runs; }

cudaError_t launch_tensor_steps(TensorPlan* p, bool src_is_a, int steps, cudaStream_t s) {
    TcParams q = p->prm[src_is_a ? 0 : 1];
    q.steps = steps;
    if (steps == 1) return launch_chained(p->kernel, dim3(p->grid), dim3(kThreads), p->smem_bytes, s, q);
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(p->grid);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = p->smem_bytes;
    cfg.stream = s;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeCooperative;
    at.val.cooperative = p->grid > 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, p->run, q);
}

}  // namespace ltl
