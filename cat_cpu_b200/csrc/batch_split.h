// batch_split.h -- host: which grids of a batch the persistent kernel (k_batch.cu) gives
// to groups of CTAs.
#pragma once

#include <algorithm>
#include <vector>

namespace ltl {

constexpr int kPersistWarps = 4;
constexpr int kPersistThreads = kPersistWarps * 32;

// Words per lane.  The shared memory of a CTA is the largest ring of any radius in the
// batch: with two words at R = 6 to 8 it would be 61 to 87 KB and leave two CTAs per SM
// to every grid of the batch (the 1024-grid ensemble of R 1..8: 61.9 ms against 48.8).
constexpr int persist_words(int R) { return R <= 5 ? 2 : 1; }

// Which grids get groups of CTAs.  Model of one generation (us) by `size` CTAs on a
// chip that holds `per_sm` CTAs on each SM: a band's rows, 0.6 of a row for each of the
// 2R+1 rows that it counts first, and a group barrier.  A row of one CTA among three or
// more per SM takes `row` times their number; the rates and rows are fitted to single
// grids at 16384^2 (k_packed_radius.cu).
struct BatchCost {
    int n, groups, R;
    double row;
    BatchCost(int n_, int nw, int R_, int per_sm) : n(n_), R(R_) {
        static const double rate[] = {1.5, 1.12, 1.0};
        const int W = n < 64 ? 1 : persist_words(R);
        groups = (nw + W - 1) / W;
        row = per_sm * rate[std::min(per_sm, 3) - 1] * (W == 2 ? 0.098 + 0.0156 * R : 0.090 + 0.0063 * R);
    }
    double start() const { return 0.6 * (2 * R + 1); }
    static constexpr double kBarrier = 1.3, kSingle = 0.3;
    double time(int size) const {
        const int lanes = size * kPersistThreads;
        const int bands = std::min(n, std::max(1, lanes / groups));
        const int turns = groups > lanes ? (groups + lanes - 1) / lanes : 1;
        return turns * row * (start() + (n + bands - 1) / bands) + (size > 1 ? kBarrier : kSingle);
    }
    // CTAs that bring a generation under t, 0 if none do
    int size_for(double t) const {
        if (time(1) <= t) return 1;
        const int b = (int)((t - kBarrier) / row - start());
        if (b < 1) return 0;
        return (int)(((long long)((n + b - 1) / b) * groups + kPersistThreads - 1) / kPersistThreads);
    }
};

// The smallest common time t for which all grids fit into `ctas` CTAs: groups side
// by side, and the sum of all CTAs' time within ctas * t.  sizes: CTAs per grid.
inline void batch_split(const std::vector<BatchCost>& grids, int ctas, std::vector<int>& sizes) {
    auto fits = [&](double t) {
        double area = 0;
        long long grouped = 0;
        for (const BatchCost& g : grids) {
            const int k = g.size_for(t);
            if (k == 0) return false;
            area += k * g.time(k);
            if (k > 1) grouped += k;
        }
        return grouped <= ctas && area <= ctas * t;
    };
    double hi = 0, lo = 0;
    for (const BatchCost& g : grids) hi += g.time(1);  // one CTA each, one after the other
    for (int i = 0; i < 24 && hi - lo > 0.01 * hi; ++i) {
        const double t = 0.5 * (lo + hi);
        (fits(t) ? hi : lo) = t;
    }
    sizes.assign(grids.size(), 1);
    for (size_t i = 0; i < grids.size(); ++i) sizes[i] = std::max(1, grids[i].size_for(hi));
}

}  // namespace ltl
