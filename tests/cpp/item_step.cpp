// Items of a problem: whole 3D nodes, at most a wave of four CTAs a
// multiprocessor, and no fewer than that or than items of item_rows.
#include <algorithm>
#include <cstdio>

#include "../../similie_b200/csrc/item_rows.cuh"

int main()
{
    for (int sms : {20, 148})
        for (int64_t item_rows : {512, 2048, 4096, 8192})
            for (int64_t side : {3, 17, 48, 64, 100, 128, 200, 256, 890}) {
                int64_t const n = std::min(3 * side * side * side, (int64_t(1) << 31) - 2);
                int64_t const step = sil::item_step(n, item_rows, sms), items = (n + step - 1) / step;
                int64_t const wave = 4 * sms;
                // an item holds up to 258 rows more than asked for (whole nodes, whole rounds of the CTA)
                int64_t const least = std::min(n / (item_rows + 258), n / (n / wave + 258));
                if (step % 3 != 0 || step < 3 || items > std::max<int64_t>(1, wave + 2) || items < least) {
                    std::printf("n %lld rows %lld sms %d: step %lld, %lld items, at least %lld\n", static_cast<long long>(n),
                                static_cast<long long>(item_rows), sms, static_cast<long long>(step),
                                static_cast<long long>(items), static_cast<long long>(least));
                    return 1;
                }
            }
    std::puts("items ok");
    return 0;
}
