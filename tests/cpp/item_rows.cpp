// The rows that the batched CG kernels read and write of an item: each of the
// item's rows once, and nothing outside it, for items anywhere below row 2^31.
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "../../similie_b200/csrc/item_rows.cuh"

static void check(int64_t begin, int64_t end)
{
    constexpr int threads = 256, U = 4;
    sil::ItemRows const rows(begin, end);
    std::vector<int> seen(static_cast<size_t>(end - begin), 0);
    char* const base = nullptr;   // of<char>(base) - base is the item's first row
    for (int tid = 0; tid < threads; ++tid) {
        auto fetch = [&](int from) {
            for (int u = 0; u < U; ++u) {
                int64_t const row = (rows.of(base) - base) + rows.ahead(from, u * threads);
                if (row < begin || row >= end) {
                    std::printf("item [%lld, %lld): reads row %lld\n", static_cast<long long>(begin),
                                static_cast<long long>(end), static_cast<long long>(row));
                    std::exit(1);
                }
            }
        };
        int row = tid;
        fetch(row);
        for (; row < rows.count; row += U * threads) {
            for (int u = 0; u < U; ++u)
                if (row + u * threads < rows.count) ++seen[static_cast<size_t>(row + u * threads)];
            fetch(row + U * threads);
        }
    }
    for (int n : seen)
        if (n != 1) {
            std::printf("item [%lld, %lld): a row taken %d times\n", static_cast<long long>(begin),
                        static_cast<long long>(end), n);
            std::exit(1);
        }
}

int main()
{
    int64_t const most = (int64_t(1) << 31) - 1;
    for (int64_t count : {1, 255, 256, 257, 1023, 1024, 1025, 4096, 5000, 3700000})
        for (int64_t end : {count, count + 12345, most - 2048, most - 1, most}) check(end - count, end);
    std::puts("rows ok");
    return 0;
}
