// The index arithmetic of the transfer kernels (cat_cpu_b200/csrc/transfer_core.cuh)
// compiled for the host (test_transfer_walk.py).
#include <cstdint>

#include <cuda_runtime.h>

template <class T>
static T __ldg(const T* p) { return *p; }
template <class T>
static T __ldcs(const T* p) { return *p; }
template <class T>
static void __stcs(T* p, T v) { *p = v; }
static inline uint32_t __funnelshift_r(uint32_t lo, uint32_t hi, uint32_t s) {
    return (uint32_t)((((uint64_t)hi << 32) | lo) >> (s & 31));
}

#include "transfer_core.cuh"

using namespace ltl;

// Items that thread `at` of `stride` visits in an array of rows x width; *sum gets
// the sum of their numbers (modulo 2^64), *last the last one's.
extern "C" long long row_walk_host(int at, int stride, int width, int rows, unsigned long long* sum, long long* last) {
    long long count = 0;
    *sum = 0;
    *last = -1;
    for (RowWalk t(at, stride, width); t.row < rows; t.next()) {
        if (t.row < 0 || t.col < 0 || t.col >= width) return -1;
        *last = (long long)t.row * width + t.col;
        *sum += (unsigned long long)*last;
        ++count;
    }
    return count;
}
