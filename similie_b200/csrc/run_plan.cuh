// run_plan.cuh -- how the marching kernels cut a column of planes into runs
// (host side, called at every launch).
#pragma once

#include <algorithm>
#include <cstdint>

namespace sil {

constexpr int kRunCandidates = 10;

// Planes per run for `columns` tiles of `length` planes over `resident` CTAs at
// a time, a run of n planes costing n + 2 steps (two of start-up): the cheapest
// total of whole waves, the longest run among equals.  Beyond eight waves of
// runs the start-up only costs more.  Among the cuts of as many waves the one
// into most runs is the cheapest, so a cut per wave count is looked at, and no
// more than kRunCandidates in all.  Host time of a call, every number of runs
// tried -> this: the 3D operator on 12x12x4000 nodes 25.9 -> 7.2 us, a 1-form
// Laplacian on 400x20x20 16.9 -> 13.5.
inline int run_length(int64_t columns, int64_t length, int64_t resident, int* looked_at = nullptr)
{
    int64_t const most = std::min(length, 8 * resident / columns + 1);
    int64_t best = length, best_cost = INT64_MAX;
    int count = 0;
    for (int64_t k = 1, runs = 0; runs < most; ++k) {
        runs = std::min(most, columns > resident ? k : k * resident / columns);
        int64_t const n = (length + runs - 1) / runs;
        int64_t const waves = (columns * ((length + n - 1) / n) + resident - 1) / resident;
        ++count;
        if (waves * (n + 2) < best_cost) {
            best_cost = waves * (n + 2);
            best = n;
        }
    }
    if (looked_at != nullptr) *looked_at = count;
    return static_cast<int>(best);
}

} // namespace sil
