// item_rows.cuh -- the rows of one work item of the batched CG kernels.
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

} // namespace sil
