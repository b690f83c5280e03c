// mag_ops.cuh -- the 2D magnetostatics residual operator at one row, shared
// by the solver and the learned preconditioner.
//
// Operator (onelab_interface/magnetostatics_onelab.hpp:1271-1426 with the
// moment stencils of magnetostatics_quantities.hpp:100-123 built at
// 1095-1258): for an interior node (i,j), over the interior sampled nodes s
// whose moment stencil touches the row, y = sum_s c(s->row) * moment(s) / mu(s);
// flat layout row = i + nx*j, identity rows on the Dirichlet boundary.
#pragma once

#include <cstdint>

namespace sil {

// `a(idx)` loads the operand at flat index idx (a pointer read, or a value
// formed on the fly, e.g. a search direction z + beta p); (i, j) are the
// row's node coordinates, row = i + nx * j.
template <class T, class A>
__device__ __forceinline__ T mag_apply_node_ij(A const& a, T const* nu, int nx, int ny, int row, int i, int j)
{
    if (i == 0 || j == 0 || i + 1 == nx || j + 1 == ny) return a(row);
    T const a0 = a(row);
    T residual = T(0);
    if (j >= 2) {
        int const s = row - nx;
        T m0 = T(0);
        m0 = m0 - a(s);
        m0 = m0 + a0;
        residual = residual + m0 * nu[s];  // c = +1
    }
    {
        T m0 = T(0);
        m0 = m0 - a0;
        m0 = m0 + a(row + nx);
        residual = residual - m0 * nu[row];  // c = -1
    }
    if (i >= 2) {
        int const s = row - 1;
        T m1 = T(0);
        m1 = m1 + a(s);
        m1 = m1 - a0;
        residual = residual - m1 * nu[s];  // c = -1
    }
    {
        T m1 = T(0);
        m1 = m1 + a0;
        m1 = m1 - a(row + 1);
        residual = residual + m1 * nu[row];  // c = +1
    }
    return residual;
}

template <class T, class A>
__device__ __forceinline__ T mag_apply_node_ld(A const& a, T const* nu, int64_t nx64, int64_t ny64, int64_t row64)
{
    // problems hold fewer than 2^31 nodes (checked by the entry points): 32-bit index arithmetic
    int const nx = static_cast<int>(nx64), ny = static_cast<int>(ny64), row = static_cast<int>(row64);
    int const j = row / nx, i = row - j * nx;
    return mag_apply_node_ij<T>(a, nu, nx, ny, row, i, j);
}

template <class T>
__device__ __forceinline__ T mag_apply_node(T const* a, T const* nu, int64_t nx64, int64_t ny64, int64_t row64)
{
    return mag_apply_node_ld<T>([a](int idx) { return a[idx]; }, nu, nx64, ny64, row64);
}

// ------------------------------------------------------------------ strips
//
// 2D strips: the 2D operator marched down a strip of columns, a warp per
// strip.  Lane l holds column c0 - 1 + l; lanes 1..30 own theirs.  Walking down
// the rows a column's operand and reluctivity at rows j - 1 and j stay in
// registers and its neighbours' come from the next lanes, so a node costs one
// load per input array where a thread per node made fourteen; four rows' loads
// are in flight before the first is used.  The values are those of
// mag_apply_node_ij (an excluded term adds a zero).
constexpr int kStripCols = 30;
constexpr int kStripBatch = 4;   // rows whose loads are issued together
constexpr int kStripWarps = 8;   // strips of a CTA

// Strips of a problem: strip w % strips of row block w / strips, `rows` rows each.
struct Strips
{
    int strips;    // per row block
    int rows;      // per strip, a multiple of kStripBatch
    int count;     // in all
    int ctas;      // of kStripWarps strips
};

__host__ __device__ inline Strips strips_of(int64_t nx, int64_t ny, int rows)
{
    Strips s {};
    s.strips = static_cast<int>((nx + kStripCols - 1) / kStripCols);
    s.rows = rows;
    s.count = s.strips * static_cast<int>((ny + rows - 1) / rows);
    s.ctas = (s.count + kStripWarps - 1) / kStripWarps;
    return s;
}

// Src: Raw load(row) and T value(Raw), the operand at a row; Own own(row), what
// only an owned row needs beside it.  out(row, q, operand, raw, own) takes the
// result of an owned row.
template <class T, class Src, class Out>
__device__ __forceinline__ void mag2d_strip(Src const& src, T const* __restrict__ nu, int nx, int ny, int c0, int j0,
                                            int j1, Out const& out)
{
    constexpr int U = kStripBatch;
    int const lane = threadIdx.x & 31, i = c0 - 1 + lane, ic = min(max(i, 0), nx - 1);
    bool const own = lane > 0 && lane <= kStripCols && i < nx, col_in = i > 0 && i + 1 < nx, left_in = i >= 2;
    auto row_of = [&](int j) { return ic + nx * min(max(j, 0), ny - 1); };
    typename Src::Raw const raw_m = src.load(row_of(j0 - 1));
    typename Src::Raw raw_c = src.load(row_of(j0));
    T n_m = nu[row_of(j0 - 1)], n_c = nu[row_of(j0)];
    T below = T(0), centre = T(0);
    bool first = true;
    for (int j = j0; j < j1; j += U) {
        typename Src::Raw raw[U];
        typename Src::Own mine[U];
        T n[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            int const at = row_of(j + 1 + u);
            raw[u] = src.load(at);
            n[u] = nu[at];
            mine[u] = src.own(row_of(j + u));
        }
        if (first) {
            below = src.value(raw_m);
            centre = src.value(raw_c);
            first = false;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            T const above = src.value(raw[u]);
            T const left = __shfl_up_sync(0xffffffffu, centre, 1), right = __shfl_down_sync(0xffffffffu, centre, 1);
            T const n_l = __shfl_up_sync(0xffffffffu, n_c, 1);
            int const jj = j + u;
            T res = T(0);
            if (jj >= 2) res = res + (centre - below) * n_m;
            res = res - (above - centre) * n_c;
            if (left_in) res = res - (left - centre) * n_l;
            res = res + (centre - right) * n_c;
            bool const in = col_in && jj > 0 && jj + 1 < ny;
            if (own && jj < j1) out(ic + nx * jj, in ? res : centre, centre, raw_c, mine[u]);
            below = centre;
            centre = above;
            raw_c = raw[u];
            n_m = n_c;
            n_c = n[u];
        }
    }
}

} // namespace sil
