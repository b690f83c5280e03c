// item_rows.cuh -- the work items of the batched CG kernels and their rows.
//
// A CTA walks its item's rows in rounds and loads the next round's while it
// works on one, clamped to the item's last row.  The rows are counted from the
// item's first, not the problem's: an item is a small part of a problem, so a
// round past its end stays within 32 bits, where a problem's own row numbers,
// accepted up to 2^31 - 1, would pass it (the last items of a problem within
// 2,000 unknowns of 2^31 looked ahead to negative rows).
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define SIL_ITEM_HD __host__ __device__ __forceinline__
#else
#define SIL_ITEM_HD inline
#endif

namespace sil {

struct ItemRows
{
    int64_t first;   // of the problem's rows
    int count;

    SIL_ITEM_HD ItemRows(int64_t begin, int64_t end) : first(begin), count(static_cast<int>(end - begin)) {}
    // The item's part of a vector of the problem.
    template <class T>
    SIL_ITEM_HD T* of(T* v) const
    {
        return v + first;
    }
    SIL_ITEM_HD int ahead(int row, int by) const
    {
        int const at = row + by;
        return at < count ? at : count - 1;
    }
};

// Unknowns of an item of a problem of n: item_rows, a whole number of 3D nodes (3
// rows each), but so many that the problem has at most one wave of four CTAs a
// multiprocessor, as every CTA sums its partials (64^3 + 80^3 + 96^3, an
// iteration: at most 592 items 62 us FP32 and 104 FP64, at most 1,024 65 and 107).
// With either gauge: four times larger items for the divergence gauge, whose apply
// is the costlier, leave 147 CTAs of 128^3 nodes (160 iterations FP64 and FP32, four
// times larger -> as here: 96^3 28.9 -> 21.9 and 19.9 -> 15.1 ms, 128^3 72 -> 53 and
// 57 -> 34, 160^3 120 -> 89 and 95 -> 60).
inline int64_t item_step(int64_t n, int64_t item_rows, int multiprocessors)
{
    constexpr int64_t threads = 256;
    int64_t const wave = (n / (4 * static_cast<int64_t>(multiprocessors)) + threads) / threads * threads;
    return (item_rows > wave ? item_rows : wave) / 3 * 3;
}

} // namespace sil
