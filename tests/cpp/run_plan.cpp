// run_length against the search over every number of runs, and how many cuts it
// looks at.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>

#include "../../similie_b200/csrc/run_plan.cuh"

static int64_t every(int64_t columns, int64_t length, int64_t resident)
{
    int64_t const most = std::min(length, 8 * resident / columns + 1);
    int64_t best = length, best_cost = INT64_MAX;
    for (int64_t runs = 1; runs <= most; ++runs) {
        int64_t const n = (length + runs - 1) / runs;
        int64_t const waves = (columns * ((length + n - 1) / n) + resident - 1) / resident;
        if (waves * (n + 2) < best_cost) {
            best_cost = waves * (n + 2);
            best = n;
        }
    }
    return best;
}

int main()
{
    std::mt19937_64 rng(1);
    auto log_uniform = [&](double hi) {
        return static_cast<int64_t>(std::exp2(std::uniform_real_distribution<double>(0.0, std::log2(hi))(rng)));
    };
    for (int i = 0; i < 200000; ++i) {
        int64_t const columns = log_uniform(100000), length = log_uniform(i % 2 != 0 ? 300 : 20000);
        for (int64_t resident : {148, 296, 444, 592}) {
            int looked = 0;
            int const n = sil::run_length(columns, length, resident, &looked);
            if (n != every(columns, length, resident) || looked > sil::kRunCandidates) {
                std::printf("columns %lld length %lld resident %lld: %d (%d cuts), %lld\n", static_cast<long long>(columns),
                            static_cast<long long>(length), static_cast<long long>(resident), n, looked,
                            static_cast<long long>(every(columns, length, resident)));
                return 1;
            }
        }
    }
    std::puts("runs ok");
    return 0;
}
