// magnetostatics.cu -- 2D and 3D linear magnetostatics on the GPU: the matrix-free residual
// operator d^T (nu d A) with identity rows on the Dirichlet boundary, and a
// batched Jacobi-preconditioned conjugate-gradient solve (FP64, or FP32
// inner sweeps inside FP64 iterative refinement).
//
// Operator (onelab_interface/magnetostatics_onelab.hpp:1271-1426 with the
// moment stencils of magnetostatics_quantities.hpp:100-123 built at
// 1095-1258): for an interior node (i,j), over the interior sampled nodes s
// whose moment stencil touches the row,
//   y = sum_s c(s->row) * moment(s) / mu(s)
// with moment0(s) = A(s+ey) - A(s) (c = +1 at s+ey, -1 at s) and
// moment1(s) = A(s) - A(s+ex) (c = -1 at s+ex, +1 at s); X moments first,
// sampled nodes in ascending flat order.  Boundary rows are the identity.
// Sampled nodes on the first row/column are excluded, as in the reference.
//
// Solver (minimize_strong_formulation_residual.hpp:1028-1304): CG from
// x = 0 with the inverse diagonal as preconditioner, stopped when
// ||r|| <= tol ||b||; the final residual is re-evaluated in FP64.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <type_traits>
#include <mutex>
#include <vector>

#include "item_rows.cuh"
#include "mag3d_march.cuh"
#include "mag_ops.cuh"
#include "precond_net.cuh"
#include "run_plan.cuh"
#include "sil_internal.cuh"

namespace sil {

namespace {

constexpr int kThreads = 256;
constexpr int kNodesPerThread = 16;
constexpr int kItemNodes = kThreads * kNodesPerThread;  // nodes per work item (one CTA)

// ------------------------------------------------------------------ operator

__global__ void mag_apply_kernel(double const* nu, double const* a, double* y, int64_t nx, int64_t ny)
{
    int64_t const row = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (row >= nx * ny) return;
    y[row] = mag_apply_node(a, nu, nx, ny, row);
}

__global__ void reciprocal_kernel(double const* mu, double* nu, int64_t n)
{
    int64_t const i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    if (i < n) nu[i] = 1.0 / mu[i];
}

// ------------------------------------------------------------------ batched CG

// Directions the flexible CG keeps at most.
constexpr int kMaxDirs = 16;

struct Item
{
    int prob;
    int index;  // item index within its problem
    int64_t begin;
    int64_t end;
};

template <class T>
struct Vecs
{
    T* x;
    T* r;
    T* z;
    T* p;
    T* q;
    T* dinv;
    T* nu;
    T* ph;  // flexible CG: m stored directions p_j at ph + j * hstride
    T* qh;  // and their images q_j = A p_j
    T* p2;  // 2D CG: the direction's second buffer (p and p2 alternate)
};

struct ProbInfo
{
    int dim;                  // 2: scalar A_z on an nx x ny grid; 3: vector A on nx x ny x nz
    int64_t nx, ny, nz;
    int64_t nodes;            // grid nodes
    int64_t n;                // unknowns: nodes (2D) or 3 * nodes (3D)
    double gamma;             // 3D gauge penalty
    int nitems;
    int first_item;
    double const* ls64[3];    // 3D: reference local spacing per axis and its inverse
    double const* ils64[3];
    float const* ls32[3];
    float const* ils32[3];
    int gauge;                // 3D: 0 penalty, 1 divergence gauge
    double const* gd64;       // divergence gauge, 8 per node: E0[3], E1[3], w, 0
    float const* gd32;
    int max_iters;            // iteration budget: the problem stops once it has done this many
    int ntiles, first_tile;   // 3D: marching tiles of the problem
};

template <class T>
__device__ __forceinline__ T const* spacing(ProbInfo const& pi, int axis)
{
    if constexpr (sizeof(T) == 8) return pi.ls64[axis];
    else return pi.ls32[axis];
}

template <class T>
__device__ __forceinline__ T const* inv_spacing(ProbInfo const& pi, int axis)
{
    if constexpr (sizeof(T) == 8) return pi.ils64[axis];
    else return pi.ils32[axis];
}

// 3D curl-curl + gauge penalty at DOF row = 3*node + c (onelab_interface/
// magnetostatics_onelab.hpp:2242-2396).  The moments are the curl
// components at the interior sampled nodes s whose stencil holds the DOF,
//   B_x(s) = A_y(s) - A_z(s) - A_y(s+z) + A_z(s+y)
//   B_y(s) = -A_x(s) + A_z(s) + A_x(s+z) - A_z(s+x)
//   B_z(s) = A_x(s) - A_y(s) - A_x(s+y) + A_y(s+x)
// (boundary DOFs dropped from the stencils), weighted by the Hodge factor of
// B (d_m / (d_a d_b), central local spacings) and 1/mu(s); the gauge term is
// gamma * (d_a d_b / d_c) * A.  Boundary rows are the identity.
template <class T>
__device__ __forceinline__ T const* gauge_table(ProbInfo const& pi)
{
    if constexpr (sizeof(T) == 8) return pi.gd64;
    else return pi.gd32;
}

// Divergence gauge.  The codifferential of the 1-form A at node m is
// (D A)(m) = sum_a E0(m, a) A_a(m) + E1(m, a) A_a(m - e_a), with the
// coefficients of boundary columns zero (they are dropped from the
// reference's stencils, magnetostatics_onelab.hpp:1894-1945).  The gauge
// term of row (n, c) is sum over the codifferential rows holding the column,
// m = n and m = n + e_c, of w(m) D(m, (n, c)) (D A)(m).
template <class T, class A>
__device__ __forceinline__ T gauge_div_ld(A const& a, T const* gd, int m, int i, int j, int k, int nx, int ny)
{
    T const* e = gd + 8 * m;
    T s = T(0);
    s = s + e[0] * a(3 * m);
    if (i > 0) s = s + e[3] * a(3 * (m - 1));
    s = s + e[1] * a(3 * m + 1);
    if (j > 0) s = s + e[4] * a(3 * (m - nx) + 1);
    s = s + e[2] * a(3 * m + 2);
    if (k > 0) s = s + e[5] * a(3 * (m - nx * ny) + 2);
    return s;
}

template <class T>
__device__ __forceinline__ T gauge_div(T const* a, T const* gd, int m, int i, int j, int k, int nx, int ny)
{
    return gauge_div_ld<T>([a](int idx) { return a[idx]; }, gd, m, i, j, k, nx, ny);
}

// Gauge term of component c at interior node n = (i, j, k), given (D A)(n).
template <class T, class A>
__device__ __forceinline__ T gauge_term_ld(A const& a, T const* gd, int n, int i, int j, int k, int nx, int ny, int c,
                                           T div_n)
{
    int const step = c == 0 ? 1 : (c == 1 ? nx : nx * ny);
    int const m = n + step;
    T const div_m = gauge_div_ld<T>(a, gd, m, i + (c == 0), j + (c == 1), k + (c == 2), nx, ny);
    T t = T(0);
    t = t + gd[8 * n + 6] * gd[8 * n + c] * div_n;
    t = t + gd[8 * m + 6] * gd[8 * m + 3 + c] * div_m;
    return t;
}

template <class T>
__device__ __forceinline__ T gauge_term(T const* a, T const* gd, int n, int i, int j, int k, int nx, int ny, int c,
                                        T div_n)
{
    int const step = c == 0 ? 1 : (c == 1 ? nx : nx * ny);
    int const m = n + step;
    T const div_m = gauge_div(a, gd, m, i + (c == 0), j + (c == 1), k + (c == 2), nx, ny);
    T t = T(0);
    t = t + gd[8 * n + 6] * gd[8 * n + c] * div_n;
    t = t + gd[8 * m + 6] * gd[8 * m + 3 + c] * div_m;
    return t;
}

// G: the divergence-gauge code is compiled in (kernels of batches that hold
// a divergence-gauge problem); without it the kernels keep the register
// budget of the penalty operator.
template <class T, bool G = false>
__device__ T mag3d_apply_row(T const* a, T const* nu, ProbInfo const& pi, int64_t row64)
{
    // fewer than 2^31 unknowns per problem (checked by the entry points)
    int const row = static_cast<int>(row64);
    int const node = row / 3;
    int const c = row - 3 * node;
    int const nx = static_cast<int>(pi.nx), ny = static_cast<int>(pi.ny), nz = static_cast<int>(pi.nz);
    int const t = node / nx, i = node - t * nx, k = t / ny, j = t - k * ny;
    auto interior = [&](int ii, int jj, int kk) {
        return ii > 0 && jj > 0 && kk > 0 && ii + 1 < nx && jj + 1 < ny && kk + 1 < nz;
    };
    if (!interior(i, j, k)) return a[row];
    int const sy = 3 * nx, sz = 3 * nx * ny;
    // A at node (i, j, k) + offset, component cc; zero on the Dirichlet boundary
    auto A = [&](int di, int dj, int dk, int cc) -> T {
        return interior(i + di, j + dj, k + dk) ? a[row - c + 3 * di + sy * dj + sz * dk + cc] : T(0);
    };
    // curl moments at the sampled node (i, j, k) + (oi, oj, ok)
    auto bx = [&](int oi, int oj, int ok) {
        T m = T(0);
        m = m + A(oi, oj, ok, 1);
        m = m - A(oi, oj, ok, 2);
        m = m - A(oi, oj, ok + 1, 1);
        m = m + A(oi, oj + 1, ok, 2);
        return m;
    };
    auto by = [&](int oi, int oj, int ok) {
        T m = T(0);
        m = m - A(oi, oj, ok, 0);
        m = m + A(oi, oj, ok, 2);
        m = m + A(oi, oj, ok + 1, 0);
        m = m - A(oi + 1, oj, ok, 2);
        return m;
    };
    auto bz = [&](int oi, int oj, int ok) {
        T m = T(0);
        m = m + A(oi, oj, ok, 0);
        m = m - A(oi, oj, ok, 1);
        m = m - A(oi, oj + 1, ok, 0);
        m = m + A(oi + 1, oj, ok, 1);
        return m;
    };
    T const* lx = spacing<T>(pi, 0);
    T const* ly = spacing<T>(pi, 1);
    T const* lz = spacing<T>(pi, 2);
    T const* ilx = inv_spacing<T>(pi, 0);
    T const* ily = inv_spacing<T>(pi, 1);
    T const* ilz = inv_spacing<T>(pi, 2);
    int const nd = node;
    auto w = [&](int oi, int oj, int ok, int m) -> T {
        T const nuv = nu[nd + oi + nx * oj + nx * ny * ok];
        if (m == 0) return lx[i + oi] * ily[j + oj] * ilz[k + ok] * nuv;
        if (m == 1) return ly[j + oj] * ilx[i + oi] * ilz[k + ok] * nuv;
        return lz[k + ok] * ilx[i + oi] * ily[j + oj] * nuv;
    };
    T res = T(0);
    T ha;
    if (c == 0) {
        res = res - w(0, 0, 0, 1) * by(0, 0, 0);
        if (interior(i, j, k - 1)) res = res + w(0, 0, -1, 1) * by(0, 0, -1);
        res = res + w(0, 0, 0, 2) * bz(0, 0, 0);
        if (interior(i, j - 1, k)) res = res - w(0, -1, 0, 2) * bz(0, -1, 0);
        ha = ly[j] * lz[k] * ilx[i];
    } else if (c == 1) {
        res = res + w(0, 0, 0, 0) * bx(0, 0, 0);
        if (interior(i, j, k - 1)) res = res - w(0, 0, -1, 0) * bx(0, 0, -1);
        res = res - w(0, 0, 0, 2) * bz(0, 0, 0);
        if (interior(i - 1, j, k)) res = res + w(-1, 0, 0, 2) * bz(-1, 0, 0);
        ha = lx[i] * lz[k] * ily[j];
    } else {
        res = res - w(0, 0, 0, 0) * bx(0, 0, 0);
        if (interior(i, j - 1, k)) res = res + w(0, -1, 0, 0) * bx(0, -1, 0);
        res = res + w(0, 0, 0, 1) * by(0, 0, 0);
        if (interior(i - 1, j, k)) res = res - w(-1, 0, 0, 1) * by(-1, 0, 0);
        ha = lx[i] * ly[j] * ilz[k];
    }
    if constexpr (G) {
        if (pi.gauge) {
            T const* gd = gauge_table<T>(pi);
            T const dn = gauge_div(a, gd, node, i, j, k, nx, ny);
            return res + static_cast<T>(pi.gamma) * gauge_term(a, gd, node, i, j, k, nx, ny, c, dn);
        }
    }
    return res + static_cast<T>(pi.gamma) * ha * a[row];
}

// The curl-curl part of the three rows of an interior node (i, j, k), from
// accessors: A(di, dj, dk, c) the 1-form at node (i, j, k) + (di, dj, dk),
// component c, zero at boundary nodes; NU(oi, oj, ok) the reluctivity at
// the sampled node (i, j, k) + (oi, oj, ok).  The curl moments shared
// between the components are formed once; each component sums its terms in
// the order of mag3d_apply_row, so the values are the same whatever the
// accessors read from.
template <class T, class AF, class NF>
__device__ __forceinline__ void mag3d_curl_rows(AF const& A, NF const& NU, ProbInfo const& pi, int i, int j, int k,
                                                T* res)
{
    int const nx = static_cast<int>(pi.nx), ny = static_cast<int>(pi.ny), nz = static_cast<int>(pi.nz);
    auto interior = [&](int ii, int jj, int kk) {
        return ii > 0 && jj > 0 && kk > 0 && ii + 1 < nx && jj + 1 < ny && kk + 1 < nz;
    };
    auto bx = [&](int oi, int oj, int ok) {
        T m = T(0);
        m = m + A(oi, oj, ok, 1);
        m = m - A(oi, oj, ok, 2);
        m = m - A(oi, oj, ok + 1, 1);
        m = m + A(oi, oj + 1, ok, 2);
        return m;
    };
    auto by = [&](int oi, int oj, int ok) {
        T m = T(0);
        m = m - A(oi, oj, ok, 0);
        m = m + A(oi, oj, ok, 2);
        m = m + A(oi, oj, ok + 1, 0);
        m = m - A(oi + 1, oj, ok, 2);
        return m;
    };
    auto bz = [&](int oi, int oj, int ok) {
        T m = T(0);
        m = m + A(oi, oj, ok, 0);
        m = m - A(oi, oj, ok, 1);
        m = m - A(oi, oj + 1, ok, 0);
        m = m + A(oi + 1, oj, ok, 1);
        return m;
    };
    T const* lx = spacing<T>(pi, 0);
    T const* ly = spacing<T>(pi, 1);
    T const* lz = spacing<T>(pi, 2);
    T const* ilx = inv_spacing<T>(pi, 0);
    T const* ily = inv_spacing<T>(pi, 1);
    T const* ilz = inv_spacing<T>(pi, 2);
    auto w = [&](int oi, int oj, int ok, int m) -> T {
        T const nuv = NU(oi, oj, ok);
        if (m == 0) return lx[i + oi] * ily[j + oj] * ilz[k + ok] * nuv;
        if (m == 1) return ly[j + oj] * ilx[i + oi] * ilz[k + ok] * nuv;
        return lz[k + ok] * ilx[i + oi] * ily[j + oj] * nuv;
    };
    bool const in_k = interior(i, j, k - 1), in_j = interior(i, j - 1, k), in_i = interior(i - 1, j, k);
    T const Bx = bx(0, 0, 0), By = by(0, 0, 0), Bz = bz(0, 0, 0);
    T const Wx = w(0, 0, 0, 0), Wy = w(0, 0, 0, 1), Wz = w(0, 0, 0, 2);
    {
        T r = T(0);
        r = r - Wy * By;
        if (in_k) r = r + w(0, 0, -1, 1) * by(0, 0, -1);
        r = r + Wz * Bz;
        if (in_j) r = r - w(0, -1, 0, 2) * bz(0, -1, 0);
        res[0] = r;
    }
    {
        T r = T(0);
        r = r + Wx * Bx;
        if (in_k) r = r - w(0, 0, -1, 0) * bx(0, 0, -1);
        r = r - Wz * Bz;
        if (in_i) r = r + w(-1, 0, 0, 2) * bz(-1, 0, 0);
        res[1] = r;
    }
    {
        T r = T(0);
        r = r - Wx * Bx;
        if (in_j) r = r + w(0, -1, 0, 0) * bx(0, -1, 0);
        r = r + Wy * By;
        if (in_i) r = r - w(-1, 0, 0, 1) * by(-1, 0, 0);
        res[2] = r;
    }
}

// Penalty gauge term of component c at node (i, j, k): gamma (d_a d_b / d_c) A_c.
template <class T>
__device__ __forceinline__ T mag3d_penalty(ProbInfo const& pi, int i, int j, int k, int c, T ac)
{
    T const g = static_cast<T>(pi.gamma);
    if (c == 0) return g * (spacing<T>(pi, 1)[j] * spacing<T>(pi, 2)[k] * inv_spacing<T>(pi, 0)[i]) * ac;
    if (c == 1) return g * (spacing<T>(pi, 0)[i] * spacing<T>(pi, 2)[k] * inv_spacing<T>(pi, 1)[j]) * ac;
    return g * (spacing<T>(pi, 0)[i] * spacing<T>(pi, 1)[j] * inv_spacing<T>(pi, 2)[k]) * ac;
}

// All three rows of an interior node at once, reading a through a loader by
// row index.  DEEP: every node of the stencil (offsets -1..1 per axis) is
// interior, so no neighbour needs the boundary test (the same values, fewer
// instructions).
template <class T, bool G, bool DEEP, class LD>
__device__ __forceinline__ void mag3d_interior_node(LD const& a, T const* nu, ProbInfo const& pi, int node, int i,
                                                    int j, int k, T* out)
{
    int const nx = static_cast<int>(pi.nx), ny = static_cast<int>(pi.ny), nz = static_cast<int>(pi.nz);
    int const row0 = 3 * node;
    auto interior = [&](int ii, int jj, int kk) {
        return DEEP || (ii > 0 && jj > 0 && kk > 0 && ii + 1 < nx && jj + 1 < ny && kk + 1 < nz);
    };
    int const sy = 3 * nx, sz = 3 * nx * ny;
    auto A = [&](int di, int dj, int dk, int cc) -> T {
        return interior(i + di, j + dj, k + dk) ? a(row0 + 3 * di + sy * dj + sz * dk + cc) : T(0);
    };
    auto NU = [&](int oi, int oj, int ok) -> T { return nu[node + oi + nx * oj + nx * ny * ok]; };
    T res[3];
    mag3d_curl_rows<T>(A, NU, pi, i, j, k, res);
    T const g = static_cast<T>(pi.gamma);
    // gauge term per component: penalty g (d_a d_b / d_c) A_c, or the divergence gauge
    T gt[3];
    bool gauge_done = false;
    if constexpr (G) {
        if (pi.gauge) {
            T const* gd = gauge_table<T>(pi);
            T const dn = gauge_div_ld<T>(a, gd, node, i, j, k, nx, ny);
            for (int c = 0; c < 3; ++c) gt[c] = g * gauge_term_ld<T>(a, gd, node, i, j, k, nx, ny, c, dn);
            gauge_done = true;
        }
    }
    if (!gauge_done)
        for (int c = 0; c < 3; ++c) gt[c] = mag3d_penalty<T>(pi, i, j, k, c, a(row0 + c));
    for (int c = 0; c < 3; ++c) out[c] = res[c] + gt[c];
}

// All three rows of a node: identity on the Dirichlet boundary, else the
// interior stencil (without boundary tests where the whole stencil is
// interior).
template <class T, bool G, class LD>
__device__ void mag3d_apply_node_ld(LD const& a, T const* nu, ProbInfo const& pi, int node, T* out)
{
    int const nx = static_cast<int>(pi.nx), ny = static_cast<int>(pi.ny), nz = static_cast<int>(pi.nz);
    int const t = node / nx, i = node - t * nx, k = t / ny, j = t - k * ny;
    if (!(i > 0 && j > 0 && k > 0 && i + 1 < nx && j + 1 < ny && k + 1 < nz)) {
        int const row0 = 3 * node;
        out[0] = a(row0);
        out[1] = a(row0 + 1);
        out[2] = a(row0 + 2);
        return;
    }
    if (i > 1 && j > 1 && k > 1 && i + 2 < nx && j + 2 < ny && k + 2 < nz)
        mag3d_interior_node<T, G, true>(a, nu, pi, node, i, j, k, out);
    else
        mag3d_interior_node<T, G, false>(a, nu, pi, node, i, j, k, out);
}

template <class T, bool G = false>
__device__ __forceinline__ void mag3d_apply_node(T const* a, T const* nu, ProbInfo const& pi, int node, T* out)
{
    mag3d_apply_node_ld<T, G>([a](int idx) { return a[idx]; }, nu, pi, node, out);
}

template <class T, bool G = false>
__device__ __forceinline__ T mag_apply_row(T const* a, T const* nu, ProbInfo const& pi, int64_t row)
{
    if (pi.dim == 2) return mag_apply_node(a, nu, pi.nx, pi.ny, row);
    return mag3d_apply_row<T, G>(a, nu, pi, row);
}

// Diagonal of the operator at a row (Jacobi preconditioner), from mu directly.
__device__ double mag_diag_row(double const* mu, ProbInfo const& pi, int64_t row)
{
    if (pi.dim == 2) {
        int64_t const i = row % pi.nx, j = row / pi.nx;
        if (i == 0 || j == 0 || i + 1 == pi.nx || j + 1 == pi.ny) return 1.0;
        double d = 0.0;
        if (j >= 2) d += 1.0 / mu[row - pi.nx];
        d += 1.0 / mu[row];
        if (i >= 2) d += 1.0 / mu[row - 1];
        d += 1.0 / mu[row];
        return d;
    }
    int64_t const node = row / 3;
    int const c = static_cast<int>(row - 3 * node);
    int64_t const nx = pi.nx, ny = pi.ny, nz = pi.nz;
    int64_t const i = node % nx, t = node / nx, j = t % ny, k = t / ny;
    auto interior = [&](int64_t ii, int64_t jj, int64_t kk) {
        return ii > 0 && jj > 0 && kk > 0 && ii + 1 < nx && jj + 1 < ny && kk + 1 < nz;
    };
    if (!interior(i, j, k)) return 1.0;
    double const* lx = pi.ls64[0];
    double const* ly = pi.ls64[1];
    double const* lz = pi.ls64[2];
    double const* ilx = pi.ils64[0];
    double const* ily = pi.ils64[1];
    double const* ilz = pi.ils64[2];
    auto w = [&](int64_t ii, int64_t jj, int64_t kk, int m) -> double {
        double const nuv = 1.0 / mu[ii + nx * (jj + ny * kk)];
        if (m == 0) return lx[ii] * ily[jj] * ilz[kk] * nuv;
        if (m == 1) return ly[jj] * ilx[ii] * ilz[kk] * nuv;
        return lz[kk] * ilx[ii] * ily[jj] * nuv;
    };
    double d = 0.0;
    if (pi.gauge) {
        // divergence gauge: sum over the codifferential rows m of w(m) D(m, row)^2
        int64_t const step = c == 0 ? 1 : (c == 1 ? nx : nx * ny);
        double const* gd = pi.gd64;
        double const e0 = gd[8 * node + c], e1 = gd[8 * (node + step) + 3 + c];
        double const gdiv = gd[8 * node + 6] * e0 * e0 + gd[8 * (node + step) + 6] * e1 * e1;
        if (c == 0) {
            d += w(i, j, k, 1) + w(i, j, k, 2);
            if (interior(i, j, k - 1)) d += w(i, j, k - 1, 1);
            if (interior(i, j - 1, k)) d += w(i, j - 1, k, 2);
        } else if (c == 1) {
            d += w(i, j, k, 0) + w(i, j, k, 2);
            if (interior(i, j, k - 1)) d += w(i, j, k - 1, 0);
            if (interior(i - 1, j, k)) d += w(i - 1, j, k, 2);
        } else {
            d += w(i, j, k, 0) + w(i, j, k, 1);
            if (interior(i, j - 1, k)) d += w(i, j - 1, k, 0);
            if (interior(i - 1, j, k)) d += w(i - 1, j, k, 1);
        }
        return d + pi.gamma * gdiv;
    }
    if (c == 0) {
        d += w(i, j, k, 1) + w(i, j, k, 2);
        if (interior(i, j, k - 1)) d += w(i, j, k - 1, 1);
        if (interior(i, j - 1, k)) d += w(i, j - 1, k, 2);
        d += pi.gamma * (ly[j] * lz[k] * ilx[i]);
    } else if (c == 1) {
        d += w(i, j, k, 0) + w(i, j, k, 2);
        if (interior(i, j, k - 1)) d += w(i, j, k - 1, 0);
        if (interior(i - 1, j, k)) d += w(i - 1, j, k, 2);
        d += pi.gamma * (lx[i] * lz[k] * ily[j]);
    } else {
        d += w(i, j, k, 0) + w(i, j, k, 1);
        if (interior(i, j - 1, k)) d += w(i, j - 1, k, 0);
        if (interior(i - 1, j, k)) d += w(i - 1, j, k, 1);
        d += pi.gamma * (lx[i] * ly[j] * ilz[k]);
    }
    return d;
}

struct Scalars
{
    double rz;        // r . z of the current iterate
    double rr;        // r . r
    double rr0;       // r . r at the start of the (inner) solve
    double inner_tol2;  // squared relative reduction the inner solve stops at
    double bb;        // b . b (outer right-hand side)
    double alpha, beta;
    double last_beta; // beta formed after the latest iteration
    double scale;     // outer residual norm used to scale the inner right-hand side
    int done;         // inner / plain solve finished
    int outer_done;   // refinement finished
    int iters;        // iterations of the current solve
    int total_iters;  // all inner iterations
    int nonfinite;
    int counter_a, counter_c;
    // flexible CG with the learned preconditioner
    double win_rr;    // r . r at the start of the stall window
    int win_iters;    // iterations into the stall window
    int fallback;     // 1: the plain solver takes over this problem
    int learned_iters;
    double pq_hist[kMaxDirs];  // p_j . q_j of the stored directions
    double coef[kMaxDirs];     // (z . q_j) / (p_j . q_j) of the current z
    // Jacobi-CG iterations (cg_begin): fields a kernel reads are never written
    // in the same kernel
    int pbuf;                  // buffer (0: p, 1: p2) holding the latest direction
    int pbuf0;                 // and at the start of the chunk
    int base_iters;            // total_iters at the start of the chunk
    int stopped[2];            // by parity of the iteration: it did not run
    double rz_it[2];           // by parity of the iteration: r . z it starts from
    double scale_prev;         // outer residual norm of the previous refinement pass
    int pending;               // 1: x still lacks alpha times the latest direction
    int cycles;                // resident solve: refinement cycles run
    int timeout;               // and 1: a wait for the group's other CTAs ran out
};

// Deterministic block sum of one double per thread.
__device__ __forceinline__ double block_sum(double v, double* smem)
{
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    int const warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    __syncthreads();
    if (lane == 0) smem[warp] = v;
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x == 0) {
        for (int w = 0; w < kThreads / 32; ++w) t += smem[w];
    }
    return t;  // valid in thread 0
}

// Last-CTA-of-the-problem reduction of K sums: every CTA publishes its
// partials (thread 0's vals) and counts in; the last CTA of the problem sums
// all partials with the whole block, in a fixed order (deterministic), and
// returns true in its thread 0 with `out` holding the K totals.
template <int K>
__device__ bool finish_reduction_k(double const* vals, double* const* parts, int item_index, int first_item, int nitems,
                                   int* counter, double* out)
{
    __shared__ int is_last;
    __shared__ double red[kThreads / 32];
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 0; k < K; ++k) parts[k][first_item + item_index] = vals[k];
        __threadfence();
        is_last = atomicAdd(counter, 1) == nitems - 1;
    }
    __syncthreads();
    if (!is_last) return false;
    __threadfence();
    for (int k = 0; k < K; ++k) {
        double v = 0.0;
        for (int j = threadIdx.x; j < nitems; j += kThreads) v += __ldcg(parts[k] + first_item + j);
        out[k] = block_sum(v, red);
    }
    if (threadIdx.x == 0) {
        *counter = 0;
        return true;
    }
    return false;
}

__device__ bool finish_reduction(double partial, double* partials, int item_index, int first_item, int nitems,
                                 int* counter, double* out)
{
    double* parts[1] = {partials};
    return finish_reduction_k<1>(&partial, parts, item_index, first_item, nitems, counter, out);
}

template <class T>
__global__ void __launch_bounds__(kThreads) cg_init_kernel(Item const* items, ProbInfo const* info, Vecs<T> const* vecs,
                                                           double const* const* rhs64, double const* const* r64,
                                                           Scalars* sc, double* part_a, double* part_b, bool from_r64)
{
    __shared__ double red[kThreads / 32];
    Item const it = items[blockIdx.x];
    Scalars* s = sc + it.prob;
    if (s->outer_done) return;
    ProbInfo const pi = info[it.prob];
    Vecs<T> const v = vecs[it.prob];
    double const scale = from_r64 ? s->scale : 1.0;
    double rz = 0.0, bb = 0.0;
    for (int64_t row = it.begin + threadIdx.x; row < it.end; row += kThreads) {
        double const b = from_r64 ? r64[it.prob][row] / scale : rhs64[it.prob][row];
        T const r = static_cast<T>(b);
        T const z = v.dinv[row] * r;
        v.x[row] = T(0);
        v.r[row] = r;
        v.z[row] = z;
        v.p[row] = z;
        rz += static_cast<double>(r) * static_cast<double>(z);
        bb += static_cast<double>(r) * static_cast<double>(r);
    }
    double const rz_b = block_sum(rz, red);
    double const bb_b = block_sum(bb, red);
    double const vals[2] = {rz_b, bb_b};
    double* parts[2] = {part_a, part_b};
    double tot[2];
    if (finish_reduction_k<2>(vals, parts, it.index, pi.first_item, pi.nitems, &s->counter_a, tot)) {
        double const trz = tot[0], tot_bb = tot[1];
        s->rz = trz;
        s->rr = tot_bb;
        s->rr0 = tot_bb;
        if (!from_r64) s->bb = tot_bb;
        s->iters = 0;
        s->done = (tot_bb == 0.0 || s->total_iters >= pi.max_iters) ? 1 : 0;
        s->nonfinite = 0;
    }
}

// ------------------------------------------------------------------ marching tiles (mag3d_march.cuh)

template <class T>
__host__ __device__ Grid3<T> march_grid(ProbInfo const& pi)
{
    Grid3<T> g {};
    g.nx = static_cast<int>(pi.nx);
    g.ny = static_cast<int>(pi.ny);
    g.nz = static_cast<int>(pi.nz);
    g.gamma = static_cast<T>(pi.gamma);
    for (int a = 0; a < 3; ++a) {
        if constexpr (sizeof(T) == 8) {
            g.l[a] = pi.ls64[a];
            g.il[a] = pi.ils64[a];
        } else {
            g.l[a] = pi.ls32[a];
            g.il[a] = pi.ils32[a];
        }
    }
    return g;
}

int march_tiles_x(ProbInfo const& pi) { return static_cast<int>((pi.nx + kMarchCols - 1) / kMarchCols); }
int march_tiles_y(ProbInfo const& pi) { return static_cast<int>((pi.ny + kMarchOwnRows - 1) / kMarchOwnRows); }

// run_length for a set of grids, once a solve: every number of runs is tried, as
// the grids' waves do not fill alike.
int march_planes(std::vector<ProbInfo> const& grids, int64_t resident)
{
    int64_t columns = 0, nz = 1;
    for (ProbInfo const& g : grids) {
        columns += static_cast<int64_t>(march_tiles_x(g)) * march_tiles_y(g);
        nz = std::max(nz, g.nz);
    }
    // beyond eight waves of runs the start-up only costs more
    int64_t const most = std::min(nz, 8 * resident / columns + 1);
    int64_t best = nz;
    double best_cost = 1e300;
    for (int64_t runs = 1; runs <= most; ++runs) {
        int64_t const z = (nz + runs - 1) / runs;
        int64_t ctas = 0;
        for (ProbInfo const& g : grids)
            ctas += static_cast<int64_t>(march_tiles_x(g)) * march_tiles_y(g) * ((g.nz + z - 1) / z);
        double const cost = static_cast<double>((ctas + resident - 1) / resident) * static_cast<double>(z + 2);
        if (cost < best_cost) {
            best_cost = cost;
            best = z;
        }
    }
    return static_cast<int>(best);
}

// A run of planes of one tile of a batched 3D problem.
struct Tile
{
    int prob;
    int index;   // tile index within its problem
    int i0, j0, k0, k1;
};

// ------------------------------------------------------------------ CG iteration
//
// One Jacobi-CG iteration is two kernels in 2D over the CTAs of the problems
// that still iterate (converged problems launch nothing), and three in 3D,
// where the direction is a pass before the apply:
//   direction  p = z + beta p_old (formed on the fly at the row and at its
//              stencil neighbours; p double-buffered), x += alpha p_old of the
//              previous iteration, q = A p, partial p.q
//   update     r -= alpha q, z = D^-1 r, partials r.z and r.r
// Chunks of iterations are captured as a CUDA graph, captured again when the
// set of iterating problems changes.
//
// No CTA waits for another one's partial: each kernel starts by summing the
// previous kernel's partials itself (every CTA of a problem the same values in
// the same order) and forms beta, the stop test or alpha from them; the
// problem's first CTA records them.  Small problems are bound by the latency of
// this chain (5.3 + 4.1 us a pair of kernels at 128^2), large ones by memory:
// at the 21 M nodes of 60 problems in FP64 the direction takes 220 us for its
// seven vectors (5.3 TB/s), the update 127 for its five (6.6 TB/s).  B200, per
// iteration of a whole solve, against partials counted in by an atomic and
// summed by the last CTA, four dependent loads of descriptors, and a thread per
// row loading its own stencil: four problems of 96^2 .. 161^2 23.1 -> 11.2 us,
// 512^2 23.3 -> 12.7, 1024^2 26.9 -> 19.8, those 60 problems 549 -> 373 (FP64)
// and 382 -> 267 (FP32).

// Everything a CTA needs to know of its item, in one 128-byte line.
template <class T>
struct alignas(128) Work
{
    T* x;
    T* r;
    T* z;
    T* p;
    T* q;
    T const* dinv;
    Scalars* s;
    double* part_pq;
    double* part_rz;
    double* part_rr;
    int begin, end;     // rows of the item
    int index;          // item (partial) number within the problem
    int npart, npq;     // partials of r.z and r.r, and of p.q
    int max_iters;
};

// Sums of two strided lists of n partials, the same in every thread of every
// CTA: thread t adds entries t, t + kThreads, ... in order, then a butterfly
// per warp, then the warps in order.
__device__ __forceinline__ void sum_partials(double const* a, double const* b, int n, double* smem, double& ta,
                                             double& tb)
{
    double va = 0.0, vb = 0.0;
    for (int j = threadIdx.x; j < n; j += kThreads) {
        va += __ldcg(a + j);
        if (b != nullptr) vb += __ldcg(b + j);
    }
    for (int o = 16; o > 0; o >>= 1) {
        va += __shfl_xor_sync(0xffffffffu, va, o);
        vb += __shfl_xor_sync(0xffffffffu, vb, o);
    }
    int const warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    if (lane == 0) {
        smem[warp] = va;
        smem[kThreads / 32 + warp] = vb;
    }
    __syncthreads();
    ta = tb = 0.0;
    for (int w = 0; w < kThreads / 32; ++w) {
        ta += smem[w];
        tb += smem[kThreads / 32 + w];
    }
}

struct Begin
{
    bool run;        // the iteration runs
    bool pending;    // x still lacks alpha p_old
    double alpha;    // of the previous iteration
    double beta;
    int pbuf;        // buffer of p_old
};

// Start of iteration c of a chunk (c > 0: completes iteration c - 1 from its
// partials).  lead: this CTA records the problem's state.  Every thread of the
// block calls it; smem holds 2 * kThreads / 32 doubles.
// in_place: the problem's directions all live in p (3D), not in p and p2 by turns.
__device__ __forceinline__ Begin cg_begin(Scalars* s, int c, double const* part_rz, double const* part_rr, int npart,
                                          int max_iters, bool lead, double* smem, bool in_place)
{
    Begin b {};
    int const now = c & 1, before = now ^ 1;
    if (s->outer_done || (c == 0 ? s->done : s->stopped[before])) {
        if (lead && threadIdx.x == 0) s->stopped[now] = 1;
        return b;
    }
    b.pbuf = in_place ? 0 : s->pbuf0 ^ now;
    if (c == 0) {
        b.run = true;
        b.beta = s->beta;
        if (lead && threadIdx.x == 0) {
            s->rz_it[0] = s->rz;
            s->stopped[0] = 0;
        }
        return b;
    }
    double const rz_old = s->rz_it[before];
    double rz = 0.0, rr = 0.0;
    sum_partials(part_rz, part_rr, npart, smem, rz, rr);
    b.pending = true;
    b.alpha = s->alpha;
    b.beta = rz / rz_old;
    bool const bad = !isfinite(rr) || !isfinite(rz);
    b.run = !(rr <= s->inner_tol2 * s->rr0 || bad || s->base_iters + c >= max_iters);
    if (lead && threadIdx.x == 0) {
        s->rz_it[now] = rz;
        s->stopped[now] = b.run ? 0 : 1;
        s->rz = rz;
        s->rr = rr;
        s->last_beta = b.beta;
        s->iters = c;
        s->total_iters = s->base_iters + c;
        s->pbuf = b.pbuf;
        s->pending = 1;
        if (bad) s->nonfinite = 1;
    }
    return b;
}

// Rows per strip: the fewest, in steps of four, at which the batch fits one
// wave of two CTAs per multiprocessor; 32 at most (a strip of R rows reads
// R + 2, and one wave of longer ones leaves too few loads in flight).
int strip_rows(std::vector<ProbInfo> const& grids)
{
    int rows = kStripBatch;
    for (; rows < 32; rows += kStripBatch) {
        int64_t ctas = 0;
        for (ProbInfo const& g : grids) ctas += strips_of(g.nx, g.ny, rows).ctas;
        if (ctas <= 2 * static_cast<int64_t>(multiprocessors())) break;
    }
    return rows;
}

// Operand z + beta p_old of the search direction, x on the side.
template <class T>
struct StripDirection
{
    struct Raw
    {
        T z, p;
    };
    using Own = T;
    T const* __restrict__ z;
    T const* __restrict__ pold;
    T const* x;
    T beta;
    bool pending;
    __device__ __forceinline__ Raw load(int row) const { return {z[row], pold[row]}; }
    __device__ __forceinline__ Own own(int row) const { return pending ? x[row] : T(0); }
    __device__ __forceinline__ T value(Raw const& r) const { return r.z + beta * r.p; }
};

// A stored operand, b on the side.
struct StripResidual
{
    using Raw = double;
    using Own = double;
    double const* __restrict__ a;
    double const* __restrict__ b;
    __device__ __forceinline__ Raw load(int row) const { return a[row]; }
    __device__ __forceinline__ Own own(int row) const { return b[row]; }
    __device__ __forceinline__ double value(Raw r) const { return r; }
};

// A CTA of strips.
template <class T>
struct alignas(16) StripWork
{
    T* x;
    T const* z;
    T* p;
    T* p2;
    T* q;
    T const* nu;
    Scalars* s;
    double* part_pq;
    double const* part_rz;
    double const* part_rr;
    int nx, ny;
    int strips, rows, count;   // Strips of the problem
    int first;                 // the CTA's first strip
    int index;                 // CTA (partial) number within the problem
    int prob;
    int npart, max_iters;
};

template <class T>
__global__ void __launch_bounds__(kThreads, 2) cg_direction2_kernel(StripWork<T> const* work, int c)
{
    __shared__ double red[2 * kThreads / 32];
    StripWork<T> const w = work[blockIdx.x];
    Begin const b = cg_begin(w.s, c, w.part_rz, w.part_rr, w.npart, w.max_iters, w.index == 0, red, false);
    if (!b.run) return;
    T* __restrict__ pnew = b.pbuf == 0 ? w.p2 : w.p;
    T* __restrict__ x = w.x;
    T* __restrict__ q = w.q;
    StripDirection<T> const src {w.z, b.pbuf == 0 ? w.p : w.p2, w.x, static_cast<T>(b.beta), b.pending};
    T const alpha = static_cast<T>(b.alpha);
    double pq = 0.0;
    int const strip = w.first + static_cast<int>(threadIdx.x) / 32;
    if (strip < w.count) {
        int const block = strip / w.strips, j0 = block * w.rows;
        mag2d_strip<T>(src, w.nu, w.nx, w.ny, (strip - block * w.strips) * kStripCols, j0, min(w.ny, j0 + w.rows),
                       [&](int row, T qr, T pr, typename StripDirection<T>::Raw const& raw, T xr) {
                           if (b.pending) x[row] = xr + alpha * raw.p;
                           pnew[row] = pr;
                           q[row] = qr;
                           pq += static_cast<double>(pr) * static_cast<double>(qr);
                       });
    }
    __syncthreads();
    double const t = block_sum(pq, red);
    if (threadIdx.x == 0) w.part_pq[w.index] = t;
}

// Z: z is stored for the 2D stencil; the 3D direction forms it again from r.
template <class T, bool Z>
__global__ void __launch_bounds__(kThreads) cg_update_kernel(Work<T> const* work, int c)
{
    __shared__ double red[2 * kThreads / 32];
    Work<T> const w = work[blockIdx.x];
    Scalars* s = w.s;
    if (s->stopped[c & 1]) return;
    ItemRows const rows(w.begin, w.end);
    T* __restrict__ r = rows.of(w.r);
    T* __restrict__ z = rows.of(w.z);
    T const* __restrict__ q = rows.of(w.q);
    T const* __restrict__ dinv = rows.of(w.dinv);
    // the first rows' loads are issued before the partials are summed
    constexpr int U = 4;
    T rv[U], qv[U], dv[U];
    int row = static_cast<int>(threadIdx.x);
    auto fetch = [&](int from) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            int const at = rows.ahead(from, u * kThreads);
            rv[u] = r[at];
            qv[u] = q[at];
            dv[u] = dinv[at];
        }
    };
    fetch(row);
    double pq, none;
    sum_partials(w.part_pq, nullptr, w.npq, red, pq, none);
    double const a = s->rz_it[c & 1] / pq;
    if (w.index == 0 && threadIdx.x == 0) {
        s->alpha = a;
        if (!isfinite(a)) s->nonfinite = 1;
    }
    T const alpha = static_cast<T>(a);
    double rz = 0.0, rr = 0.0;
    for (; row < rows.count; row += U * kThreads) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            if (row + u * kThreads >= rows.count) continue;
            T const rn = rv[u] - alpha * qv[u], zn = dv[u] * rn;
            r[row + u * kThreads] = rn;
            if constexpr (Z) z[row + u * kThreads] = zn;
            rz += static_cast<double>(rn) * static_cast<double>(zn);
            rr += static_cast<double>(rn) * static_cast<double>(rn);
        }
        fetch(row + U * kThreads);
    }
    __syncthreads();
    double const rz_b = block_sum(rz, red), rr_b = block_sum(rr, red);
    if (threadIdx.x == 0) {
        w.part_rz[w.index] = rz_b;
        w.part_rr[w.index] = rr_b;
    }
}

// End of a chunk of `c` iterations: completes the last one (one CTA per item;
// only each problem's first works).
template <class T, bool IN_PLACE>
__global__ void __launch_bounds__(kThreads) cg_close_kernel(Work<T> const* work, int c)
{
    __shared__ double red[2 * kThreads / 32];
    Work<T> const w = work[blockIdx.x];
    if (w.index != 0) return;
    Begin const b = cg_begin(w.s, c, w.part_rz, w.part_rr, w.npart, w.max_iters, true, red, IN_PLACE);
    __syncthreads();
    if (threadIdx.x == 0 && !w.s->outer_done) {
        w.s->done = b.run ? 0 : 1;
        w.s->beta = w.s->last_beta;
    }
}

// 3D problems: p = D^-1 r + beta p in place and x += alpha p_old as a pass of
// their own, then the apply.  z is not stored and p not double-buffered, so an
// iteration of a medium batch stays in L2: at the 4.9 M rows of 64^3 + 80^3 + 96^3
// in FP32 its six vectors are 118 MB, with z and the second p 157.  Forming the
// direction inside the marching apply (between its copies and its planes) moves
// two vectors less but costs more instructions than this pass costs memory: one
// 160^3 problem, per iteration, FP64 292 -> 265 us, FP32 217 -> 157.  Bound by
// memory (6.4 TB/s at 160^3 in FP64); two rows in flight a thread instead of
// four cost 8% of an FP64 iteration.
template <class T>
__global__ void __launch_bounds__(kThreads) cg_direction3_kernel(Work<T> const* work, int c)
{
    __shared__ double red[2 * kThreads / 32];
    Work<T> const w = work[blockIdx.x];
    ItemRows const rows(w.begin, w.end);
    T const* __restrict__ r = rows.of(w.r);
    T const* __restrict__ dinv = rows.of(w.dinv);
    T* __restrict__ x = rows.of(w.x);
    T* __restrict__ p = rows.of(w.p);
    // the first rows are on their way while the partials are summed
    constexpr int U = 4;
    T rv[U], dv[U], xv[U], pv[U];
    int row = static_cast<int>(threadIdx.x);
    auto fetch = [&](int from) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            int const at = rows.ahead(from, u * kThreads);
            rv[u] = r[at];
            dv[u] = dinv[at];
            xv[u] = x[at];
            pv[u] = p[at];
        }
    };
    fetch(row);
    Begin const b = cg_begin(w.s, c, w.part_rz, w.part_rr, w.npart, w.max_iters, w.index == 0, red, true);
    if (!b.run) return;
    T const beta = static_cast<T>(b.beta), alpha = static_cast<T>(b.alpha);
    for (; row < rows.count; row += U * kThreads) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            int const at = row + u * kThreads;
            if (at >= rows.count) continue;
            p[at] = dv[u] * rv[u] + beta * pv[u];
            if (b.pending) x[at] = xv[u] + alpha * pv[u];
        }
        fetch(row + U * kThreads);
    }
}

// q = A p and the partials of p.q for batches of penalty-gauge problems, in
// marching tiles (mag3d_march.cuh).
template <class T>
__global__ void __launch_bounds__(kMarchThreads, 4)
        cg_march_kernel(Tile const* tiles, int const* act, ProbInfo const* info, Vecs<T> const* vecs, Scalars const* sc,
                        double* part_pq, int c)
{
    __shared__ MarchSmem<T> sm;
    __shared__ double red[kThreads / 32];
    static_assert(kMarchThreads == kThreads, "block_sum covers the block");
    Tile const t = tiles[act[blockIdx.x]];
    Scalars const* s = sc + t.prob;
    if (s->stopped[c & 1]) return;
    ProbInfo const& pi = info[t.prob];
    Vecs<T> const v = vecs[t.prob];
    T const* p = v.p;
    double pq = 0.0;
    mag3d_march(sm, march_grid<T>(pi), static_cast<T const*>(v.nu), p, t.i0, t.j0, t.k0, t.k1, [&](int row, T q, T pv) {
        v.q[row] = q;
        pq += static_cast<double>(pv) * static_cast<double>(q);
    });
    double const pq_b = block_sum(pq, red);
    if (threadIdx.x == 0) part_pq[pi.first_tile + t.index] = pq_b;
}

// The apply of batches with the divergence gauge, whose stencil reaches two
// nodes: a thread per node.
template <class T>
__global__ void __launch_bounds__(kThreads) cg_apply3_kernel(Item const* items, int const* act, ProbInfo const* info,
                                                             Vecs<T> const* vecs, Scalars const* sc, double* part_pq,
                                                             int c)
{
    __shared__ double red[kThreads / 32];
    Item const it = items[act[blockIdx.x]];
    Scalars const* s = sc + it.prob;
    if (s->stopped[c & 1]) return;
    ProbInfo const pi = info[it.prob];
    Vecs<T> const v = vecs[it.prob];
    T const* p = v.p;
    double pq = 0.0;
    for (int64_t node = it.begin / 3 + threadIdx.x; node < it.end / 3; node += kThreads) {
        T q[3];
        mag3d_apply_node<T, true>(p, v.nu, pi, static_cast<int>(node), q);
        for (int cc = 0; cc < 3; ++cc) {
            int const row = static_cast<int>(3 * node + cc);
            v.q[row] = q[cc];
            pq += static_cast<double>(p[row]) * static_cast<double>(q[cc]);
        }
    }
    double const pq_b = block_sum(pq, red);
    if (threadIdx.x == 0) part_pq[pi.first_item + it.index] = pq_b;
}

// Start or continue the CG of a refinement pass on the new outer residual:
// r = r64 / scale, z = D^-1 r, x = 0 (the correction restarts; x64 holds the
// previous ones), r.z and r.r.  fresh: p_old = z and beta = 0, so the first
// direction is z.  Otherwise the direction of the previous pass is kept (the
// Krylov space survives the residual replacement).  The pass ended at
// iterate k with (r.z)_k and beta_old = (r.z)_k / (r.z)_{k-1}; the replaced
// residual continues iterate k, so its direction is z + beta' p_{k-1} with
// beta' = (r.z)~ / (r.z)_{k-1}, all in the units of the new scale: p_{k-1}
// is rho p_old there and (r.z)_{k-1} is rho^2 (r.z)_k / beta_old, rho =
// scale_prev / scale, so beta = beta_old (r.z)~ / (rho (r.z)_k) applied to
// the stored p_old.
//
// That holds while the recurrence follows the true residual.  On a grid so
// small or thin that CG reaches the precision of T within a pass, the recurrence
// goes on falling after the true residual has stopped; the replaced residual is
// then nothing the stored direction was built for, beta' grows without bound
// and every later direction is the old one (FP32, 3x70 nodes: 2e-7 after 3,000
// iterations, 3x4: a residual of 1e32).  follows() tells such a pass, after which
// the direction restarts from z, by a true r.z a hundred times the recurrence's
// (ten times its residual).  The thin grids then converge to 1e-10 within 600
// iterations; 228 solves of 24^2 .. 1024^2, in both precisions, and in 3D of 16^3
// .. 80^3, keep every bit.
constexpr double kLostRz = 100.0;
__device__ __forceinline__ bool follows(double rz_true, double scale, double rz_rec, double scale_prev)
{
    double const rho = scale_prev / scale;
    return rz_true <= kLostRz * (rho * rho * rz_rec);
}

template <class T>
__global__ void __launch_bounds__(kThreads) cg_replace_kernel(Item const* items, int const* act, ProbInfo const* info,
                                                              Vecs<T> const* vecs, double const* const* r64,
                                                              Scalars* sc, double* part_a, double* part_b, int fresh)
{
    __shared__ double red[kThreads / 32];
    Item const it = items[act[blockIdx.x]];
    Scalars* s = sc + it.prob;
    if (s->outer_done) return;
    ProbInfo const pi = info[it.prob];
    Vecs<T> const v = vecs[it.prob];
    double const scale = s->scale;
    ItemRows const rows(it.begin, it.end);
    double const* __restrict__ src = rows.of(r64[it.prob]);
    T const* __restrict__ dinv = rows.of(v.dinv);
    T* __restrict__ x = rows.of(v.x);
    T* __restrict__ rv = rows.of(v.r);
    T* __restrict__ zv = rows.of(v.z);
    T* __restrict__ pold = rows.of(s->pbuf == 0 ? v.p : v.p2);
    double rz = 0.0, rr = 0.0;
#pragma unroll 4
    for (int row = static_cast<int>(threadIdx.x); row < rows.count; row += kThreads) {
        T const r = static_cast<T>(src[row] / scale);
        T const z = dinv[row] * r;
        x[row] = T(0);
        rv[row] = r;
        zv[row] = z;
        if (fresh) pold[row] = z;
        rz += static_cast<double>(r) * static_cast<double>(z);
        rr += static_cast<double>(r) * static_cast<double>(r);
    }
    double const rz_b = block_sum(rz, red);
    double const rr_b = block_sum(rr, red);
    double const vals[2] = {rz_b, rr_b};
    double* parts[2] = {part_a, part_b};
    double tot[2];
    if (finish_reduction_k<2>(vals, parts, it.index, pi.first_item, pi.nitems, &s->counter_a, tot)) {
        double const trz = tot[0], tot_rr = tot[1];
        // beta = 0 (the direction restarts from z) on a fresh pass, when no
        // iterate has run since the last replacement, and when the recurrence
        // has lost the residual
        bool const keep = !fresh && s->iters > 0 && s->rz > 0.0 && s->scale_prev > 0.0
                          && follows(trz, scale, s->rz, s->scale_prev);
        s->beta = keep ? s->beta * trz / ((s->scale_prev / scale) * s->rz) : 0.0;
        if (fresh) s->pbuf = 0;
        s->pbuf0 = s->pbuf;
        s->base_iters = s->total_iters;
        s->pending = 0;
        s->rz = trz;
        s->rr = tot_rr;
        s->rr0 = tot_rr;
        s->iters = 0;
        s->done = (tot_rr == 0.0 || s->total_iters >= pi.max_iters) ? 1 : 0;
        s->nonfinite = 0;
    }
}

// ------------------------------------------------------------------ flexible CG (learned preconditioner)
//
// Notay's truncated flexible CG, FCG(m): z = M(r) from the learned
// preconditioner, which is not a fixed linear operator, is made A-orthogonal
// to the last m directions, p = z - sum_j (z.q_j)/(p_j.q_j) p_j with
// q_j = A p_j, then alpha = (p.r)/(p.q).  Directions live in a ring of m
// slots; iteration k writes slot k mod m.  m = 1 is the one-step truncation
// p = z + beta p.  A problem whose residual has not dropped 10x over `window`
// iterations is marked for the plain solver.

// x = 0, r = r64 / scale (precision T), rr0 = r.r; stall window reset.
// Problems already handed to the plain solver get a zero correction.  After
// the first pass (fresh = 0) the stored directions are kept: the projections
// (z.q_j)/(p_j.q_j) p_j and alpha = (p.r)/(p.q) do not depend on the units
// the directions were formed in, so the flexible CG continues on the
// replaced residual instead of restarting.
template <class T>
__global__ void __launch_bounds__(kThreads) fcg_init_kernel(Item const* items, int const* act, ProbInfo const* info,
                                                            Vecs<T> const* vecs, double const* const* r64,
                                                            Scalars* sc, double* part, int fresh)
{
    __shared__ double red[kThreads / 32];
    Item const it = items[act != nullptr ? act[blockIdx.x] : blockIdx.x];
    Scalars* s = sc + it.prob;
    if (s->outer_done) return;
    Vecs<T> const v = vecs[it.prob];
    if (s->fallback) {
        for (int64_t row = it.begin + threadIdx.x; row < it.end; row += kThreads) v.x[row] = T(0);
        return;
    }
    ProbInfo const pi = info[it.prob];
    double const scale = s->scale;
    double rr = 0.0;
    for (int64_t row = it.begin + threadIdx.x; row < it.end; row += kThreads) {
        T const r = static_cast<T>(r64[it.prob][row] / scale);
        v.x[row] = T(0);
        v.r[row] = r;
        rr += static_cast<double>(r) * static_cast<double>(r);
    }
    double const rr_b = block_sum(rr, red);
    double tot = 0.0;
    if (finish_reduction(rr_b, part, it.index, pi.first_item, pi.nitems, &s->counter_a, &tot)) {
        s->rr = tot;
        s->rr0 = tot;
        s->win_rr = tot;
        s->win_iters = 0;
        if (fresh) s->iters = 0;
        s->done = (tot == 0.0 || s->total_iters >= pi.max_iters) ? 1 : 0;
        s->nonfinite = 0;
    }
}

// Sums over a problem's CTAs of the K values each thread holds.  A CTA's sums go
// to parts[k * stride + index]; the last of the problem's n CTAs to count in
// adds the partials, a warp per value, in a fixed order, and returns true in
// thread 0 with the totals in `out` (shared).  (With a block-wide sum per value
// at both ends the eight of fcg_orth_kernel took half of its 33 us.)
template <int K>
__device__ __forceinline__ bool fcg_sums(double (&v)[K], double* parts, int64_t stride, int index, int n, int* counter,
                                         double (&red)[K][kThreads / 32], double (&out)[K])
{
    __shared__ int is_last;
    int const warp = threadIdx.x / 32, lane = threadIdx.x % 32;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        for (int o = 16; o > 0; o >>= 1) v[k] += __shfl_xor_sync(0xffffffffu, v[k], o);
        if (lane == 0) red[k][warp] = v[k];
    }
    __syncthreads();
    if (warp == 0) {
        if (lane < K) {
            double t = 0.0;
            for (int w = 0; w < kThreads / 32; ++w) t += red[lane][w];
            __stcg(parts + lane * stride + index, t);
            __threadfence();
        }
        __syncwarp();
        if (lane == 0) is_last = atomicAdd(counter, 1) == n - 1;
    }
    __syncthreads();
    if (!is_last) return false;
    __threadfence();
    for (int k = warp; k < K; k += kThreads / 32) {
        double t = 0.0;
#pragma unroll 4
        for (int j = lane; j < n; j += 32) t += __ldcg(parts + k * stride + j);
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0) out[k] = t;
    }
    __syncthreads();
    if (threadIdx.x != 0) return false;
    *counter = 0;
    return true;
}

// Partials z.q_j over the stored directions (the first min(iters, m)); the
// last CTA forms coef_j = (z.q_j)/(p_j.q_j).  M >= m is the compile-time bound.
template <class T, int M>
__global__ void __launch_bounds__(kThreads) fcg_orth_kernel(Item const* items, int const* act, ProbInfo const* info,
                                                            Vecs<T> const* vecs, Scalars* sc, double* parts_base,
                                                            int64_t hstride, int m, int nitems_all)
{
    __shared__ double red[M][kThreads / 32];
    __shared__ double tot[M];
    Item const it = items[act != nullptr ? act[blockIdx.x] : blockIdx.x];
    Scalars* s = sc + it.prob;
    if (s->done || s->outer_done || s->fallback) return;
    ProbInfo const pi = info[it.prob];
    Vecs<T> const v = vecs[it.prob];
    int const nvalid = min(s->iters, m);
    if (nvalid == 0) return;
    T const* __restrict__ z = v.z;
    T const* __restrict__ qh = v.qh;
    int const end = static_cast<int>(it.end);
    double acc[M];
#pragma unroll
    for (int j = 0; j < M; ++j) acc[j] = 0.0;
#pragma unroll 2
    for (int row = static_cast<int>(it.begin) + threadIdx.x; row < end; row += kThreads) {
        double const zr = static_cast<double>(z[row]);
#pragma unroll
        for (int j = 0; j < M; ++j)
            if (j < nvalid) acc[j] += zr * static_cast<double>(qh[j * hstride + row]);
    }
    if (fcg_sums<M>(acc, parts_base + pi.first_item, nitems_all, it.index, pi.nitems, &s->counter_a, red, tot)) {
        for (int j = 0; j < nvalid; ++j) {
            s->coef[j] = tot[j] / s->pq_hist[j];
            if (!isfinite(s->coef[j])) s->nonfinite = 1;
        }
    }
}

// p_slot = z - sum_j coef_j p_j, slot = iters mod m.  When the ring is full
// the slot being written is also the oldest term of the sum; each thread
// reads its element of every p_j before writing.
template <class T, int M>
__global__ void __launch_bounds__(kThreads) fcg_direction_kernel(Item const* items, int const* act, Vecs<T> const* vecs,
                                                                 Scalars const* sc, int64_t hstride, int m)
{
    Item const it = items[act != nullptr ? act[blockIdx.x] : blockIdx.x];
    Scalars const* s = sc + it.prob;
    if (s->done || s->outer_done || s->fallback) return;
    Vecs<T> const v = vecs[it.prob];
    int const nvalid = min(s->iters, m);
    int const slot = s->iters % m;
    T c[M];
#pragma unroll
    for (int j = 0; j < M; ++j) c[j] = j < nvalid ? static_cast<T>(s->coef[j]) : T(0);
    T const* __restrict__ z = v.z;
    T* ph = v.ph;
    int const end = static_cast<int>(it.end);
    // the rows' loads go out in batches: a row's store may not wait for the next row's loads
    constexpr int U = M > 8 ? 1 : 2;
    for (int row = static_cast<int>(it.begin) + threadIdx.x; row < end; row += U * kThreads) {
        T p[U], h[U][M];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            int const at = min(row + u * kThreads, end - 1);
            p[u] = z[at];
#pragma unroll
            for (int j = 0; j < M; ++j) h[u][j] = j < nvalid ? ph[j * hstride + at] : T(0);
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
#pragma unroll
            for (int j = 0; j < M; ++j)
                if (j < nvalid) p[u] -= c[j] * h[u][j];
            if (row + u * kThreads < end) ph[slot * hstride + row + u * kThreads] = p[u];
        }
    }
}

// The direction p_slot as a strip's operand, r on the side.
template <class T>
struct StripSlot
{
    using Raw = T;
    using Own = T;
    T const* __restrict__ p;
    T const* __restrict__ r;
    __device__ __forceinline__ Raw load(int row) const { return p[row]; }
    __device__ __forceinline__ Own own(int row) const { return r[row]; }
    __device__ __forceinline__ T value(Raw v) const { return v; }
};

// q_slot = A p_slot in strips, partials p.q and p.r; the last CTA stores p.q
// for the slot and forms alpha.
template <class T>
__global__ void __launch_bounds__(kThreads) fcg_apply_kernel(StripWork<T> const* work, Vecs<T> const* vecs, int64_t hstride,
                                                             int m, int64_t part_stride)
{
    __shared__ double red[2][kThreads / 32];
    __shared__ double tot[2];
    StripWork<T> const w = work[blockIdx.x];
    Scalars* s = w.s;
    if (s->done || s->outer_done || s->fallback) return;
    Vecs<T> const v = vecs[w.prob];
    int const slot = s->iters % m;
    T* __restrict__ q = v.qh + slot * hstride;
    double sums[2] = {0.0, 0.0};
    int const strip = w.first + static_cast<int>(threadIdx.x) / 32;
    if (strip < w.count) {
        int const block = strip / w.strips, j0 = block * w.rows;
        mag2d_strip<T>(StripSlot<T> {v.ph + slot * hstride, v.r}, w.nu, w.nx, w.ny, (strip - block * w.strips) * kStripCols,
                       j0, min(w.ny, j0 + w.rows), [&](int row, T qr, T p, T, T r) {
                           q[row] = qr;
                           sums[0] += static_cast<double>(p) * static_cast<double>(qr);
                           sums[1] += static_cast<double>(p) * static_cast<double>(r);
                       });
    }
    int const ctas = (w.count + kThreads / 32 - 1) / (kThreads / 32);
    if (fcg_sums<2>(sums, w.part_pq, part_stride, w.index, ctas, &s->counter_a, red, tot)) {
        s->pq_hist[slot] = tot[0];
        s->alpha = tot[1] / tot[0];
        if (!isfinite(s->alpha)) s->nonfinite = 1;
    }
}

// x += alpha p_slot, r -= alpha q_slot, partial r.r; the last CTA advances
// the iteration (and so the slot), checks convergence and the stall window, and
// switches the problem off for the network (`active`) once it stops.
template <class T>
__global__ void __launch_bounds__(kThreads) fcg_update_kernel(Item const* items, int const* act, ProbInfo const* info,
                                                              Vecs<T> const* vecs, Scalars* sc, double* part,
                                                              int window, int64_t hstride, int m, int* active)
{
    __shared__ double red[1][kThreads / 32];
    __shared__ double total[1];
    Item const it = items[act != nullptr ? act[blockIdx.x] : blockIdx.x];
    Scalars* s = sc + it.prob;
    if (s->done || s->outer_done || s->fallback) return;
    ProbInfo const pi = info[it.prob];
    Vecs<T> const v = vecs[it.prob];
    int const slot = s->iters % m;
    T const* __restrict__ p = v.ph + slot * hstride;
    T const* __restrict__ q = v.qh + slot * hstride;
    T* __restrict__ rv = v.r;
    T* __restrict__ xv = v.x;
    T const alpha = static_cast<T>(s->alpha);
    int const end = static_cast<int>(it.end);
    double rr[1] = {0.0};
#pragma unroll 4
    for (int row = static_cast<int>(it.begin) + threadIdx.x; row < end; row += kThreads) {
        T const r = rv[row] - alpha * q[row];
        xv[row] = xv[row] + alpha * p[row];
        rv[row] = r;
        rr[0] += static_cast<double>(r) * static_cast<double>(r);
    }
    if (fcg_sums<1>(rr, part + pi.first_item, 0, it.index, pi.nitems, &s->counter_c, red, total)) {
        double const tot = total[0];
        s->rr = tot;
        s->iters += 1;
        s->total_iters += 1;
        s->learned_iters += 1;
        if (!isfinite(tot)) s->nonfinite = 1;
        if (tot <= s->inner_tol2 * s->rr0 || s->nonfinite || s->total_iters >= pi.max_iters) s->done = 1;
        if (++s->win_iters >= window) {
            if (!(tot <= 0.01 * s->win_rr)) {
                s->fallback = 1;
                s->done = 1;
            }
            s->win_rr = tot;
            s->win_iters = 0;
        }
        if (s->done) active[it.prob] = 0;
    }
}

// active[p] = 1 while problem p's flexible CG still iterates; the network
// skips the others.
__global__ void fcg_active_kernel(Scalars const* sc, int np, int* active)
{
    int const p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= np) return;
    Scalars const& s = sc[p];
    active[p] = (s.done || s.outer_done || s.fallback) ? 0 : 1;
}

// State of a problem after its outer residual's |r|^2 = tot.
__device__ __forceinline__ void residual_done(Scalars* s, double tot, double tol2, double floor2, int mark)
{
    s->rr = tot;
    s->scale_prev = s->scale;
    s->scale = sqrt(tot);
    if (mark && (tot <= tol2 * s->bb || !isfinite(tot))) s->outer_done = 1;
    // Next inner solve: reduce the (unit-scaled) residual until the outer
    // residual would be half the tolerance, but never below the floor the
    // inner precision can reach.
    s->inner_tol2 = fmax(floor2, 0.25 * tol2 * s->bb / fmax(tot, 1e-300));
    if (!isfinite(tot)) s->nonfinite = 1;
}

// r64 = b - A x64 and its norm (outer residual, FP64); marks outer convergence.
// act: the items to visit (NULL: every item, one CTA each).
template <bool G = false>
__global__ void __launch_bounds__(kThreads) residual64_kernel(Item const* items, int const* act, ProbInfo const* info,
                                                              double const* const* nu64, double const* const* rhs,
                                                              double* const* x64, double* const* r64, Scalars* sc,
                                                              double* part, double tol2, double floor2, int mark)
{
    __shared__ double red[kThreads / 32];
    Item const it = items[act != nullptr ? act[blockIdx.x] : blockIdx.x];
    Scalars* s = sc + it.prob;
    if (s->outer_done) return;
    ProbInfo const pi = info[it.prob];
    double rr = 0.0;
    if (pi.dim == 3) {
        for (int64_t node = it.begin / 3 + threadIdx.x; node < it.end / 3; node += kThreads) {
            double ax[3];
            mag3d_apply_node<double, G>(x64[it.prob], nu64[it.prob], pi, static_cast<int>(node), ax);
            for (int c = 0; c < 3; ++c) {
                double const r = rhs[it.prob][3 * node + c] - ax[c];
                r64[it.prob][3 * node + c] = r;
                rr += r * r;
            }
        }
    } else {
        for (int64_t row = it.begin + threadIdx.x; row < it.end; row += kThreads) {
            double const ax = mag_apply_row<double, G>(x64[it.prob], nu64[it.prob], pi, row);
            double const r = rhs[it.prob][row] - ax;
            r64[it.prob][row] = r;
            rr += r * r;
        }
    }
    double const rr_b = block_sum(rr, red);
    double tot = 0.0;
    if (finish_reduction(rr_b, part, it.index, pi.first_item, pi.nitems, &s->counter_a, &tot))
        residual_done(s, tot, tol2, floor2, mark);
}

// The same for 2D batches, in strips.
template <class T>
__global__ void __launch_bounds__(kThreads, 2)
        residual64_strip_kernel(StripWork<T> const* work, double const* const* nu64, double const* const* rhs,
                                double* const* x64, double* const* r64, double tol2, double floor2, int mark)
{
    __shared__ double red[kThreads / 32];
    StripWork<T> const w = work[blockIdx.x];
    Scalars* s = w.s;
    if (s->outer_done) return;
    double* r64p = r64[w.prob];
    double rr = 0.0;
    int const strip = w.first + static_cast<int>(threadIdx.x) / 32;
    if (strip < w.count) {
        int const block = strip / w.strips, j0 = block * w.rows;
        mag2d_strip<double>(StripResidual {x64[w.prob], rhs[w.prob]}, nu64[w.prob], w.nx, w.ny,
                            (strip - block * w.strips) * kStripCols, j0, min(w.ny, j0 + w.rows),
                            [&](int row, double ax, double, double, double b) {
                                double const r = b - ax;
                                r64p[row] = r;
                                rr += r * r;
                            });
    }
    double const rr_b = block_sum(rr, red);
    double tot = 0.0;
    int const ctas = (w.count + kThreads / 32 - 1) / (kThreads / 32);
    if (finish_reduction(rr_b, w.part_pq, w.index, 0, ctas, &s->counter_a, &tot))
        residual_done(s, tot, tol2, floor2, mark);
}

// The same for batches of 3D penalty-gauge problems, in marching tiles.
__global__ void __launch_bounds__(kMarchThreads, 4)
        residual64_march_kernel(Tile const* tiles, int const* act, ProbInfo const* info, double const* const* nu64,
                                double const* const* rhs, double* const* x64, double* const* r64, Scalars* sc,
                                double* part, double tol2, double floor2, int mark)
{
    __shared__ MarchSmem<double> sm;
    __shared__ double red[kThreads / 32];
    Tile const t = tiles[act[blockIdx.x]];
    Scalars* s = sc + t.prob;
    if (s->outer_done) return;
    ProbInfo const& pi = info[t.prob];
    double const* b = rhs[t.prob];
    double* r64p = r64[t.prob];
    double rr = 0.0;
    mag3d_march(sm, march_grid<double>(pi), nu64[t.prob], static_cast<double const*>(x64[t.prob]), t.i0, t.j0, t.k0, t.k1,
                [&](int row, double ax, double) {
                    double const r = b[row] - ax;
                    r64p[row] = r;
                    rr += r * r;
                });
    double const rr_b = block_sum(rr, red);
    double tot = 0.0;
    if (finish_reduction(rr_b, part, t.index, pi.first_tile, pi.ntiles, &s->counter_a, &tot))
        residual_done(s, tot, tol2, floor2, mark);
}

// x64 += scale * e (inner correction, promoted to FP64).
template <class T>
__global__ void __launch_bounds__(kThreads) refine_kernel(Item const* items, int const* act, Vecs<T> const* vecs,
                                                          double* const* x64, Scalars const* sc)
{
    Item const it = items[act != nullptr ? act[blockIdx.x] : blockIdx.x];
    Scalars const* s = sc + it.prob;
    if (s->outer_done) return;
    ItemRows const rows(it.begin, it.end);
    T const* __restrict__ e = rows.of(vecs[it.prob].x);
    double* __restrict__ x = rows.of(x64[it.prob]);
    double const scale = s->scale;
    if (s->pending) {
        // the last iteration's step is still to be added to x
        T const* __restrict__ p = rows.of(s->pbuf == 0 ? vecs[it.prob].p : vecs[it.prob].p2);
        T const alpha = static_cast<T>(s->alpha);
#pragma unroll 4
        for (int row = static_cast<int>(threadIdx.x); row < rows.count; row += kThreads)
            x[row] += scale * static_cast<double>(e[row] + alpha * p[row]);
        return;
    }
#pragma unroll 4
    for (int row = static_cast<int>(threadIdx.x); row < rows.count; row += kThreads)
        x[row] += scale * static_cast<double>(e[row]);
}

// nu = 1/mu per node (FP64 and, for the inner solve, the precision T) and
// the inverse diagonal of the operator per unknown.
template <class T>
__global__ void setup_kernel(Item const* items, ProbInfo const* info, double const* const* mu, double* const* nu64,
                             Vecs<T> const* vecs)
{
    Item const it = items[blockIdx.x];
    ProbInfo const pi = info[it.prob];
    Vecs<T> const v = vecs[it.prob];
    double const* m = mu[it.prob];
    int const per_node = pi.dim == 2 ? 1 : 3;
    for (int64_t row = it.begin + threadIdx.x; row < it.end; row += kThreads) {
        if (row % per_node == 0) {
            int64_t const node = row / per_node;
            double const nu = 1.0 / m[node];
            nu64[it.prob][node] = nu;
            v.nu[node] = static_cast<T>(nu);
        }
        v.dinv[row] = static_cast<T>(1.0 / mag_diag_row(m, pi, row));
    }
}

__global__ void copy_kernel(Item const* items, double const* const* src, double* const* dst, Scalars const* sc)
{
    Item const it = items[blockIdx.x];
    (void)sc;
    for (int64_t row = it.begin + threadIdx.x; row < it.end; row += kThreads) dst[it.prob][row] = src[it.prob][row];
}

// ------------------------------------------------------------------ resident solve (2D)
//
// The whole refinement loop of a 2D problem in one cooperative launch, its
// vectors on chip: a group of CTAs, one per multiprocessor, holds consecutive
// grid rows each, p, nu and D^-1 in shared memory and r, x and q in registers,
// so an iteration reads nothing from memory but the two neighbour rows of z
// and the group's partial sums.  An iteration has two waits for the group (after
// p.q and after r.z), where its sums pass through global memory; a group whose
// problem has ended leaves, and groups of several problems run side by side.  The
// arithmetic is the launch-per-kernel path's, the sums in another order.
//
// B200, per iteration against two kernels: four problems of 96^2 .. 161^2 11.2 ->
// 6.2 us, 512^2 12.7 -> 7.2, 1024^2 19.8 -> 12.5 (FP64), six problems of 128^2 ..
// 1024^2 41 -> 28, sixty 373 -> 237 (FP64) and 267 -> 137 (FP32).  What bounds it
// is waiting, in the two meetings (about 1.7 us each at sixteen CTAs) and at the
// barriers between the loops: two thirds of the stalls at 128^2 and half at
// 1024^2, where the shared-memory reads of 7,168 nodes keep their pipe busy for
// 35 % of the time.
//
// A launch that the device refuses, and a group of which a wait ran out, leave
// their problems to the kernels per iteration.
constexpr int kResThreads = 512;
// Nodes of a thread at most (r, x and q take three registers of T each): 7,168
// a CTA in FP64, 14,336 in FP32.
template <class T>
constexpr int kResMaxPerThread = sizeof(T) == 8 ? 14 : 28;
constexpr int kResPollLimit = 1 << 22;                    // polls of a wait before it gives up (seconds)

struct ResidentCta
{
    int prob;
    int g, group;      // CTA number within the problem's group, and the group's size
    int ja, jb;        // owned rows
    int nx, ny;
    int slots;         // first mail slot of the group
};

// A group meets by mail: each CTA stores its two sums into its own pair of
// slots and polls everybody's, so the data is its own arrival flag and a
// meeting costs one trip through L2 after the last arrival (a counter and then
// the sums would cost two, and all arrivals queue on the counter).  An empty
// slot holds a NaN no sum is stored as.  Meetings use four sets of slots in
// turn; a CTA empties its slots of meeting k + 2 after passing meeting k - 1,
// when everyone has read what they held (meeting k - 2).  Of two meetings in a
// row at least one carries data, and its release and acquire order the emptying
// before anyone's poll of meeting k + 2.
constexpr unsigned long long kNoMail = 0x7ff8decafc0ffee1ull;
constexpr int kMailSets = 4;
constexpr int kMailPerLane = 8;   // of a polling lane: groups of up to 256 CTAs
constexpr int kHaloAhead = 2;   // halo nodes per row that a thread loads ahead

// RELEASE: what the CTA stored before is visible to whoever reads the mail.
template <bool RELEASE>
__device__ __forceinline__ void mail_store(unsigned long long* slot, double v)
{
    unsigned long long w = static_cast<unsigned long long>(__double_as_longlong(v));
    if (w == kNoMail) w = 0x7ff8000000000000ull;
    if constexpr (RELEASE) asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(slot), "l"(w) : "memory");
    else asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(slot), "l"(w) : "memory");
}
__device__ __forceinline__ unsigned long long mail_load(unsigned long long const* slot)
{
    unsigned long long w;
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(w) : "l"(slot) : "memory");
    return w;
}

// M: nodes of a thread.  Local node n = tid + m * kResThreads; the arrays are
// padded to M * kResThreads nodes, whose r and q are zero, so the loops load
// without a guard.
template <class T, int M>
__global__ void __launch_bounds__(kResThreads, 1)
        cg_resident_kernel(ResidentCta const* ctas, Vecs<T> const* vecs, double const* const* nu64,
                           double const* const* rhs, double* const* x64, double* const* r64, Scalars* sc,
                           unsigned long long* mail, double tol2, int max_iter, int spent, int chunk, int poll_limit)
{
    constexpr int kNodes = M * kResThreads;
    extern __shared__ __align__(16) unsigned char res_smem[];
    __shared__ double red[2][kResThreads / 32];
    __shared__ double sums[2];
    __shared__ int aborted;
    ResidentCta const c = ctas[blockIdx.x];
    Scalars* s = sc + c.prob;
    if (s->outer_done) return;   // the whole group's
    int const tid = threadIdx.x, nx = c.nx, ny = c.ny, rows = c.jb - c.ja, count = rows * nx;
    int64_t const first = static_cast<int64_t>(c.ja) * nx;   // global row number of local node 0
    T* ps = reinterpret_cast<T*>(res_smem);                  // rows ja-1 .. jb (and padding)
    T* ns = ps + kNodes + 2 * nx;                            // rows ja-1 .. jb-1
    T* ds = ns + kNodes + nx;                                // rows ja .. jb-1
    Vecs<T> const v = vecs[c.prob];
    unsigned long long* const box = mail + c.slots;          // [set][CTA][2]
    int meeting = 0;
    if (tid == 0) aborted = 0;

    // The group's sums of a and, with `data`, of b over all threads, the same
    // bits in every CTA; with `data` what the CTAs stored to global memory before
    // is visible after.  False when a wait ran out.
    auto meet = [&](auto data, double a, double b, double& sum_a, double& sum_b) -> bool {
        constexpr bool kData = decltype(data)::value, kBoth = kData;
        for (int o = 16; o > 0; o >>= 1) {
            a += __shfl_xor_sync(0xffffffffu, a, o);
            b += __shfl_xor_sync(0xffffffffu, b, o);
        }
        if ((tid & 31) == 0) {
            red[0][tid >> 5] = a;
            red[1][tid >> 5] = b;
        }
        __syncthreads();
        if (tid < 32) {
            double ta = tid < kResThreads / 32 ? red[0][tid & 15] : 0.0, tb = tid < kResThreads / 32 ? red[1][tid & 15] : 0.0;
            for (int o = 8; o > 0; o >>= 1) {
                ta += __shfl_xor_sync(0xffffffffu, ta, o);
                tb += __shfl_xor_sync(0xffffffffu, tb, o);
            }
            unsigned long long* const now = box + static_cast<int64_t>(meeting & (kMailSets - 1)) * 2 * c.group;
            unsigned long long* const later = box + static_cast<int64_t>((meeting + 2) & (kMailSets - 1)) * 2 * c.group;
            if (tid < 2) {
                later[2 * c.g + tid] = kNoMail;
                if (kBoth || tid == 0) mail_store<kData>(now + 2 * c.g + tid, tid == 0 ? ta : tb);
            }
            // this lane's share of the mail, all of it asked for at once
            unsigned long long wa[kMailPerLane], wb[kMailPerLane];
            int tries = 0;
            bool lost = poll_limit == 0, waiting = !lost;
#pragma unroll
            for (int u = 0; u < kMailPerLane; ++u) wa[u] = wb[u] = tid + 32 * u < c.group ? kNoMail : 0ull;
            while (waiting) {
                waiting = false;
#pragma unroll
                for (int u = 0; u < kMailPerLane; ++u) {
                    unsigned long long const* slot = now + 2 * (tid + 32 * u);
                    if (wa[u] == kNoMail) wa[u] = mail_load(slot);
                    if (kBoth && wb[u] == kNoMail) wb[u] = mail_load(slot + 1);
                }
#pragma unroll
                for (int u = 0; u < kMailPerLane; ++u) waiting = waiting || wa[u] == kNoMail || (kBoth && wb[u] == kNoMail);
                if (waiting && ++tries >= poll_limit) {
                    lost = true;
                    break;
                }
            }
            double va = 0.0, vb = 0.0;
#pragma unroll
            for (int u = 0; u < kMailPerLane; ++u) {
                va += __longlong_as_double(static_cast<long long>(wa[u]));
                if (kBoth) vb += __longlong_as_double(static_cast<long long>(wb[u]));
            }
            if constexpr (kData) asm volatile("fence.acq_rel.gpu;" ::: "memory");
            if (__any_sync(0xffffffffu, lost)) {
                if (tid == 0) {
                    aborted = 1;
                    s->timeout = 1;
                }
            }
            for (int o = 16; o > 0; o >>= 1) {
                va += __shfl_xor_sync(0xffffffffu, va, o);
                vb += __shfl_xor_sync(0xffffffffu, vb, o);
            }
            if (tid == 0) {
                sums[0] = va;
                sums[1] = vb;
            }
        }
        ++meeting;
        __syncthreads();
        sum_a = sums[0];
        sum_b = sums[1];
        return aborted == 0;
    };

    // which of this thread's nodes are interior, and which lie in a row that
    // another CTA reads
    unsigned inner = 0, edge = 0;
#pragma unroll 1
    for (int m = 0; m < M; ++m) {
        int const n = tid + m * kResThreads;
        if (n >= count) continue;
        int const jl = n / nx, i = n - jl * nx, j = c.ja + jl;
        if (i > 0 && i + 1 < nx && j > 0 && j + 1 < ny) inner |= 1u << m;
        if (jl == 0 || jl == rows - 1) edge |= 1u << m;
    }
    auto is = [](unsigned mask, int m) { return ((mask >> m) & 1u) != 0; };
    bool const lower = c.ja > 0, upper = c.jb < ny;
    // The reluctivity of the first row and column is zero here: it only enters
    // the terms that the operator leaves out, which so add a zero.
    for (int n = tid; n < kNodes + nx; n += kResThreads) {
        int const jl = n / nx, i = n - jl * nx, j = c.ja - 1 + jl;
        ns[n] = j > 0 && i > 0 && j < c.jb ? v.nu[first - nx + n] : T(0);
    }
    for (int n = tid; n < kNodes; n += kResThreads) ds[n] = n < count ? v.dinv[first + n] : T(0);
    for (int n = tid; n < kNodes + 2 * nx; n += kResThreads) ps[n] = T(0);
    double const* const nu = nu64[c.prob] + first;
    double const* const b = rhs[c.prob] + first;
    double* const xg = x64[c.prob] + first;
    double* const rg = r64[c.prob] + first;
    T* const zg = v.z + first;

    double const bb = s->bb;
    double scale = s->scale, beta_last = 0.0, rz_cur = 0.0, none;
    int total_iters = s->total_iters, iters = 0, cycles = 0, nonfinite = 0, outer = 0;
    bool ok = true;
    T r[M], x[M], q[M];
    __syncthreads();
    while (true) {
        // r64 = b - A x64, its norm
        double acc = 0.0;
#pragma unroll 1
        for (int n = tid, m = 0; n < count; n += kResThreads, ++m) {
            double const a0 = __ldcg(xg + n);
            double ax = a0;
            if (is(inner, m)) {
                int const jl = n / nx, i = n - jl * nx, j = c.ja + jl;
                ax = 0.0;
                if (j >= 2) ax = ax + (a0 - __ldcg(xg + n - nx)) * nu[n - nx];
                ax = ax - (__ldcg(xg + n + nx) - a0) * nu[n];
                if (i >= 2) ax = ax - (__ldcg(xg + n - 1) - a0) * nu[n - 1];
                ax = ax + (a0 - __ldcg(xg + n + 1)) * nu[n];
            }
            double const res = b[n] - ax;
            rg[n] = res;
            acc += res * res;
        }
        double tot;
        if (!(ok = meet(std::false_type {}, acc, 0.0, tot, none))) break;
        double const scale_prev = scale;
        scale = sqrt(tot);
        if (!isfinite(tot)) nonfinite = 1;
        if (tot <= tol2 * bb || !isfinite(tot)) {
            outer = 1;
            break;
        }
        // the batch's budget, of which an earlier stage has used `spent`
        if (spent + static_cast<int64_t>(cycles) * chunk >= max_iter) break;
        double const inner_tol2 = 0.25 * tol2 * bb / fmax(tot, 1e-300);
        // residual replacement (cg_replace_kernel)
        double rz = 0.0, rr = 0.0;
#pragma unroll
        for (int m = 0; m < M; ++m) {
            int const n = tid + m * kResThreads;
            T const rn = n < count ? static_cast<T>(rg[n] / scale) : T(0), z = ds[n] * rn;
            r[m] = rn;
            x[m] = T(0);
            if (is(edge, m)) __stcg(zg + n, z);
            rz += static_cast<double>(rn) * static_cast<double>(z);
            rr += static_cast<double>(rn) * static_cast<double>(rn);
        }
        double rz0, rr0;
        if (!(ok = meet(std::true_type {}, rz, rr, rz0, rr0))) break;
        bool const keep = cycles > 0 && iters > 0 && rz_cur > 0.0 && scale_prev > 0.0
                          && follows(rz0, scale, rz_cur, scale_prev);
        double beta = keep ? beta_last * rz0 / ((scale_prev / scale) * rz_cur) : 0.0;
        rz_cur = rz0;
        iters = 0;
        nonfinite = 0;
        bool done = rr0 == 0.0 || total_iters >= max_iter;
        T alpha = T(0);   // of the step x still lacks
        for (int it = 0; it < chunk && !done; ++it) {
            // p = z + beta p (and the previous step's x += alpha p), halo rows
            // too: their z is on its way while the own nodes are formed
            T const bt = static_cast<T>(beta);
            T zl[kHaloAhead], zu[kHaloAhead];
#pragma unroll
            for (int h = 0; h < kHaloAhead; ++h) {
                int const i = min(tid + h * kResThreads, nx - 1);
                zl[h] = lower ? __ldcg(zg - nx + i) : T(0);
                zu[h] = upper ? __ldcg(zg + count + i) : T(0);
            }
#pragma unroll
            for (int m = 0; m < M; ++m) {
                int const n = tid + m * kResThreads;
                T const po = ps[n + nx];
                x[m] = x[m] + alpha * po;
                if (n < count) ps[n + nx] = ds[n] * r[m] + bt * po;
            }
#pragma unroll
            for (int h = 0; h < kHaloAhead; ++h) {
                int const i = tid + h * kResThreads;
                if (i < nx) {
                    if (lower) ps[i] = zl[h] + bt * ps[i];
                    if (upper) ps[count + nx + i] = zu[h] + bt * ps[count + nx + i];
                }
            }
            for (int i = tid + kHaloAhead * kResThreads; i < nx; i += kResThreads) {
                if (lower) ps[i] = __ldcg(zg - nx + i) + bt * ps[i];
                if (upper) ps[count + nx + i] = __ldcg(zg + count + i) + bt * ps[count + nx + i];
            }
            __syncthreads();
            double pq = 0.0;
#pragma unroll
            for (int m = 0; m < M; ++m) {
                int const n = tid + m * kResThreads;
                T const* p = ps + n + nx;
                T const a0 = n < count ? p[0] : T(0), nc = ns[n + nx];
                T qv = T(0);
                qv = qv + (a0 - p[-nx]) * ns[n];
                qv = qv - (p[nx] - a0) * nc;
                qv = qv - (p[-1] - a0) * ns[n + nx - 1];
                qv = qv + (a0 - p[1]) * nc;
                qv = is(inner, m) ? qv : a0;
                q[m] = qv;
                pq += static_cast<double>(a0) * static_cast<double>(qv);
            }
            double tpq;
            if (!(ok = meet(std::false_type {}, pq, 0.0, tpq, none))) break;
            double const a = rz_cur / tpq;
            alpha = static_cast<T>(a);
            rz = rr = 0.0;
#pragma unroll
            for (int m = 0; m < M; ++m) {
                int const n = tid + m * kResThreads;
                T const rn = r[m] - alpha * q[m], z = ds[n] * rn;
                r[m] = rn;
                if (is(edge, m)) __stcg(zg + n, z);
                rz += static_cast<double>(rn) * static_cast<double>(z);
                rr += static_cast<double>(rn) * static_cast<double>(rn);
            }
            double rz1, rr1;
            if (!(ok = meet(std::true_type {}, rz, rr, rz1, rr1))) break;
            beta = beta_last = rz1 / rz_cur;
            rz_cur = rz1;
            ++iters;
            ++total_iters;
            bool const bad = !isfinite(rr1) || !isfinite(rz1) || !isfinite(a);
            if (bad) nonfinite = 1;
            done = rr1 <= inner_tol2 * rr0 || bad || total_iters >= max_iter;
        }
        if (!ok) break;
        // x64 += scale x
#pragma unroll
        for (int m = 0; m < M; ++m) {
            int const n = tid + m * kResThreads;
            if (n < count)
                __stcg(xg + n, __ldcg(xg + n) + scale * static_cast<double>(x[m] + alpha * ps[n + nx]));
        }
        if (!(ok = meet(std::true_type {}, 0.0, 0.0, none, none))) break;
        ++cycles;
    }
    if (c.g == 0 && tid == 0) {
        s->scale = scale;
        s->total_iters = total_iters;
        s->iters = iters;
        s->nonfinite = nonfinite;
        s->outer_done = outer;
        s->cycles = cycles;
    }
}

// ------------------------------------------------------------------ host driver

struct DeviceBuffer
{
    void* ptr = nullptr;
    ~DeviceBuffer() { cudaFree(ptr); }
};

// Memory of small solves comes from a pool of the device that keeps up to
// kPoolKeep bytes between calls (the rest goes back to the device at the next
// synchronisation, and all of it when a larger solve finds no memory).  The pool
// is stream-ordered, so threads and streams can share it.  cudaMalloc and
// cudaFree map and unmap at every call, 0.4 ms each: four 2D problems of 96^2 ..
// 161^2 5.4 -> 4.6 ms a solve, one 32^3 5.4 -> 4.7.  Larger solves, of whose time
// that is a percent or two, do not hold on to memory.
constexpr size_t kPoolKeep = size_t(64) << 20;

cudaMemPool_t solve_pool()
{
    static std::mutex mutex;
    static cudaMemPool_t pools[16] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev >= 16) return nullptr;
    std::lock_guard<std::mutex> lock(mutex);
    if (pools[dev] == nullptr) {
        cudaMemPoolProps props {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t pool = nullptr;
        if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) {
            cudaGetLastError();
            return nullptr;
        }
        uint64_t keep = kPoolKeep;
        cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
        pools[dev] = pool;
    }
    return pools[dev];
}

struct SolveBuffer
{
    void* ptr = nullptr;
    cudaStream_t stream = nullptr;
    bool pooled = false;

    cudaError_t take(size_t bytes, cudaStream_t st)
    {
        stream = st;
        cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
        cudaMemPool_t pool = nullptr;
        if (cudaStreamIsCapturing(st, &capture) == cudaSuccess && capture == cudaStreamCaptureStatusNone) pool = solve_pool();
        if (pool != nullptr && bytes <= kPoolKeep) {
            pooled = cudaMallocFromPoolAsync(&ptr, bytes, pool, st) == cudaSuccess;
            if (pooled) return cudaSuccess;
            cudaGetLastError();
            ptr = nullptr;
        }
        cudaError_t e = cudaMalloc(&ptr, bytes);
        if (e == cudaErrorMemoryAllocation && pool != nullptr) {
            cudaGetLastError();
            cudaMemPoolTrimTo(pool, 0);
            e = cudaMalloc(&ptr, bytes);
        }
        return e;
    }
    ~SolveBuffer()
    {
        if (pooled) {
            cudaStreamSynchronize(stream);   // as cudaFree: nothing of the call runs on
            cudaFreeAsync(ptr, stream);
        } else cudaFree(ptr);
    }
};

// One problem of a batch, 2D or 3D, as the solver driver sees it.
struct ProblemDesc
{
    int dim;
    int64_t nx, ny, nz;
    double gamma;
    double const* node_mu;
    double const* rhs;
    double* solution;
    double const* coords[3];  // 3D: host node coordinates per axis
    int gauge = 0;            // 3D: 0 penalty, 1 divergence gauge
};

// Central local spacing of a node along one axis (one-sided at the ends),
// the length SimiLie's magnetostatics operator uses for its Hodge factors
// (onelab_interface/magnetostatics_onelab.hpp:856-870).
double local_spacing(double const* c, int64_t n, int64_t i)
{
    if (n < 2) return 1.0;
    if (i == 0) return c[1] - c[0];
    if (i + 1 == n) return c[n - 1] - c[n - 2];
    return 0.5 * (c[i + 1] - c[i - 1]);
}

// ---- divergence gauge: the codifferential's coefficients, read off the
// library's own codifferential (the reference's SimiLie Codifferential::value
// at every node, identity metric, node positions) applied to six probes.
// Probe (a, parity) is 1 on component a at the interior nodes whose index
// along a has that parity; at a node of the same parity the output is the
// coefficient of A_a(m), at the others that of A_a(m - e_a), each already
// zero where the column is a boundary DOF.

__global__ void gauge_probe_kernel(double* p, int nx, int ny, int nz, int a, int parity)
{
    int64_t const node = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (node >= static_cast<int64_t>(nx) * ny * nz) return;
    int const i = static_cast<int>(node % nx);
    int64_t const t = node / nx;
    int const j = static_cast<int>(t % ny), k = static_cast<int>(t / ny);
    int const idx = a == 0 ? i : (a == 1 ? j : k);
    bool const in = i > 0 && j > 0 && k > 0 && i + 1 < nx && j + 1 < ny && k + 1 < nz;
    for (int c = 0; c < 3; ++c) p[3 * node + c] = (c == a && in && idx % 2 == parity) ? 1.0 : 0.0;
}

__global__ void gauge_extract_kernel(double const* q, double* gd, int nx, int ny, int nz, int a, int parity)
{
    int64_t const node = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (node >= static_cast<int64_t>(nx) * ny * nz) return;
    int const i = static_cast<int>(node % nx);
    int64_t const t = node / nx;
    int const j = static_cast<int>(t % ny), k = static_cast<int>(t / ny);
    int const idx = a == 0 ? i : (a == 1 ? j : k);
    if (idx % 2 == parity) gd[8 * node + a] = q[node];
    else gd[8 * node + 3 + a] = q[node];
}

// w(m) = product of the local spacings (the reference's codifferential
// weights, magnetostatics_onelab.hpp:1896-1898); FP32 copy of the table.
__global__ void gauge_weight_kernel(ProbInfo pi, double* gd, float* gd32)
{
    int64_t const node = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (node >= pi.nodes) return;
    int64_t const i = node % pi.nx, t = node / pi.nx, j = t % pi.ny, k = t / pi.ny;
    gd[8 * node + 6] = pi.ls64[0][i] * pi.ls64[1][j] * pi.ls64[2][k];
    gd[8 * node + 7] = 0.0;
    if (gd32 != nullptr)
        for (int q = 0; q < 8; ++q) gd32[8 * node + q] = static_cast<float>(gd[8 * node + q]);
}

// gd (8 doubles per node), gd32 (8 floats per node, may be NULL); probe (3
// doubles per node) and out (1 per node) are scratch.  pi carries the
// device spacing tables.
sil_status build_divergence_gauge(ProblemDesc const& q, ProbInfo const& pi, double* gd, float* gd32, double* probe,
                                  double* out, cudaStream_t st)
{
    int64_t const len[3] = {q.nx, q.ny, q.nz};
    sil_geometry geo = nullptr;
    if (sil_status s = sil_geometry_create(&geo, 3, q.coords, len, nullptr); s != SIL_OK) return s;
    struct GeoGuard
    {
        sil_geometry g;
        ~GeoGuard() { sil_geometry_destroy(g); }
    } guard {geo};
    sil_field in {}, o {};
    in.data = probe;
    in.dtype = SIL_F64;
    in.ndims = 3;
    in.ncomp = 3;
    o.data = out;
    o.dtype = SIL_F64;
    o.ndims = 3;
    o.ncomp = 1;
    int64_t stride = 1;
    for (int a = 0; a < 3; ++a) {
        in.extent[a] = o.extent[a] = len[a];
        in.stride[a] = 3 * stride;  // solver layout: 3 * (i + nx (j + ny k)) + c
        o.stride[a] = stride;
        stride *= len[a];
    }
    in.comp_stride = 1;
    o.comp_stride = 1;
    int const nodes_blocks = static_cast<int>((pi.nodes + 255) / 256);
    int const nx = static_cast<int>(q.nx), ny = static_cast<int>(q.ny), nz = static_cast<int>(q.nz);
    SIL_CUDA_CHECK(cudaMemsetAsync(gd, 0, sizeof(double) * 8 * pi.nodes, st));
    for (int a = 0; a < 3; ++a)
        for (int parity = 0; parity < 2; ++parity) {
            gauge_probe_kernel<<<nodes_blocks, 256, 0, st>>>(probe, nx, ny, nz, a, parity);
            if (sil_status s = sil_codifferential(geo, st, 7u, 1, &in, &o); s != SIL_OK) return s;
            gauge_extract_kernel<<<nodes_blocks, 256, 0, st>>>(out, gd, nx, ny, nz, a, parity);
        }
    gauge_weight_kernel<<<nodes_blocks, 256, 0, st>>>(pi, gd, gd32);
    SIL_CUDA_CHECK(cudaGetLastError());
    return SIL_OK;
}

// Dynamic shared memory of the resident kernel at most: the 227 KB a CTA can
// have less its static part.  Every launch allows its instance this much: the
// attribute belongs to the kernel and the device, not to the call, so a smaller
// value of one host thread would refuse another's launch of the same instance.
constexpr size_t kResSmemMost = 226 * 1024;

// Shared memory of the resident kernel with m nodes per thread, and the rows a
// CTA can hold of an nx-wide grid.
template <class T>
size_t resident_smem(int m, int64_t nx)
{
    return (3 * static_cast<size_t>(m) * kResThreads + 3 * static_cast<size_t>(nx)) * sizeof(T);
}
template <class T>
int64_t resident_rows(int64_t nx)
{
    return resident_smem<T>(kResMaxPerThread<T>, nx) <= kResSmemMost ? kResThreads * kResMaxPerThread<T> / nx : 0;
}

// The kernel's instances by nodes per thread.
template <class T>
int resident_nodes(int per_thread)
{
    for (int m : {2, 4, 8, 14})
        if (per_thread <= m) return m;
    return kResMaxPerThread<T>;
}

// CTAs a 2D problem needs to be resident (0: it does not fit the GPU).
template <class T>
int resident_ctas(ProblemDesc const& q, int sms)
{
    if (q.dim != 2 || q.nx * q.ny > static_cast<int64_t>(sms) * kResThreads * kResMaxPerThread<T>) return 0;
    int64_t const rows = resident_rows<T>(q.nx);
    if (rows < 1) return 0;
    int64_t const g = (q.ny + rows - 1) / rows;
    return g <= sms ? static_cast<int>(g) : 0;
}

// One cooperative launch: problems side by side, one CTA per multiprocessor.
struct ResidentWave
{
    std::vector<int> probs;
    std::vector<ResidentCta> ctas;
    size_t smem = 0;
    int per_thread = 0;   // nodes of a thread: the kernel's instance
};

// Nodes per CTA below which another CTA in the group costs more in meetings
// than it saves: 8 sqrt(nodes), 1,024 at least.  Measured per FP64 iteration:
// 64^2 with 1,024 nodes a CTA 3.6 us, with 2,048 4.6; 128^2 1,024 4.7, 2,048 4.4,
// 4,096 5.7; 256^2 1,024 5.7, 2,048 5.3, 4,096 5.8; 512^2 1,771 8.2, 4,096 6.4.
int64_t resident_enough(ProblemDesc const& q)
{
    return std::max<int64_t>(1024, static_cast<int64_t>(8.0 * std::sqrt(static_cast<double>(q.nx * q.ny))));
}

// Problems into waves (largest first, each into the first wave with room), then
// a wave's spare CTAs to the problems with the most nodes per CTA.
template <class T>
std::vector<ResidentWave> plan_resident(std::vector<ProblemDesc> const& probs, int sms)
{
    std::vector<ResidentWave> waves;
    std::vector<int> order, need(probs.size(), 0), room;
    for (size_t p = 0; p < probs.size(); ++p) {
        need[p] = resident_ctas<T>(probs[p], sms);
        if (need[p] > 0) order.push_back(static_cast<int>(p));
    }
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) {
        return probs[a].nx * probs[a].ny > probs[b].nx * probs[b].ny;
    });
    for (int p : order) {
        size_t w = 0;
        while (w < waves.size() && room[w] < need[p]) ++w;
        if (w == waves.size()) {
            waves.emplace_back();
            room.push_back(sms);
        }
        waves[w].probs.push_back(p);
        room[w] -= need[p];
    }
    int slots = 0;
    for (size_t w = 0; w < waves.size(); ++w) {
        ResidentWave& wave = waves[w];
        std::vector<int64_t> g;
        int64_t widest = 0;
        for (int p : wave.probs) g.push_back(need[p]);
        for (int spare = room[w]; spare > 0; --spare) {
            int64_t most = 0;
            size_t at = g.size();
            for (size_t k = 0; k < g.size(); ++k) {
                ProblemDesc const& q = probs[wave.probs[k]];
                int64_t const nodes = (q.ny + g[k] - 1) / g[k] * q.nx;
                if (g[k] < q.ny && nodes > resident_enough(q) && nodes > most) {
                    most = nodes;
                    at = k;
                }
            }
            if (at == g.size()) break;
            ++g[at];
        }
        for (size_t k = 0; k < g.size(); ++k) {
            int const p = wave.probs[k];
            int const nx = static_cast<int>(probs[p].nx), ny = static_cast<int>(probs[p].ny);
            int const rows = static_cast<int>((ny + g[k] - 1) / g[k]), group = (ny + rows - 1) / rows;
            for (int i = 0; i < group; ++i)
                wave.ctas.push_back({p, i, group, i * rows, std::min(ny, (i + 1) * rows), nx, ny, slots});
            slots += 2 * kMailSets * group;
            widest = std::max<int64_t>(widest, nx);
            wave.per_thread = std::max(wave.per_thread, (rows * nx + kResThreads - 1) / kResThreads);
        }
        wave.per_thread = resident_nodes<T>(wave.per_thread);
        wave.smem = resident_smem<T>(wave.per_thread, widest);
    }
    return waves;
}

template <class T>
void const* resident_kernel(int per_thread)
{
    switch (per_thread) {
    case 2: return reinterpret_cast<void const*>(cg_resident_kernel<T, 2>);
    case 4: return reinterpret_cast<void const*>(cg_resident_kernel<T, 4>);
    case 8: return reinterpret_cast<void const*>(cg_resident_kernel<T, 8>);
    case 14: return reinterpret_cast<void const*>(cg_resident_kernel<T, 14>);
    default: return reinterpret_cast<void const*>(cg_resident_kernel<T, kResMaxPerThread<T>>);
    }
}

// Blocks the resident solve may take: one per multiprocessor, or the caller's
// limit (a lane polls kMailPerLane of a group's slots).
int chip_blocks(sil_chip_limits const& limits)
{
    return limits.blocks < 0 ? multiprocessors() : std::min(limits.blocks, 32 * kMailPerLane);
}

template <class T>
sil_status solve_batch_rows(std::vector<ProblemDesc> const& probs, sil_solve_settings const& set,
                            sil_solve_diagnostics* diag, cudaStream_t stream, nn::Net* learned,
                            sil_chip_limits& limits, int item_rows)
{
    int const np = static_cast<int>(probs.size());
    // Work items: contiguous row ranges of each problem (item_step), one CTA each.
    std::vector<Item> items;
    std::vector<ProbInfo> info(np);
    int64_t total_rows = 0;
    // 3D spacing tables, per problem [ls_x ls_y ls_z ils_x ils_y ils_z].
    std::vector<double> sp64;
    std::vector<int64_t> sp_off(np, -1);
    for (int p = 0; p < np; ++p) {
        ProblemDesc const& q = probs[p];
        ProbInfo& pi = info[p];
        pi = ProbInfo {};
        pi.dim = q.dim;
        pi.nx = q.nx;
        pi.ny = q.ny;
        pi.nz = q.dim == 3 ? q.nz : 1;
        pi.nodes = pi.nx * pi.ny * pi.nz;
        pi.n = q.dim == 3 ? 3 * pi.nodes : pi.nodes;
        pi.gamma = q.gamma;
        pi.max_iters = set.max_iterations > 0 ? set.max_iterations : 100000;
        pi.first_item = static_cast<int>(items.size());
        int idx = 0;
        int64_t const step = item_step(pi.n, item_rows, multiprocessors());
        for (int64_t b = 0; b < pi.n; b += step, ++idx) items.push_back({p, idx, b, std::min(pi.n, b + step)});
        pi.nitems = idx;
        total_rows += pi.n;
        if (q.dim == 3) {
            sp_off[p] = static_cast<int64_t>(sp64.size());
            int64_t const len[3] = {q.nx, q.ny, q.nz};
            for (int a = 0; a < 3; ++a)
                for (int64_t i = 0; i < len[a]; ++i) sp64.push_back(local_spacing(q.coords[a], len[a], i));
            for (int a = 0; a < 3; ++a)
                for (int64_t i = 0; i < len[a]; ++i) sp64.push_back(1.0 / local_spacing(q.coords[a], len[a], i));
        }
    }
    std::vector<float> sp32(sp64.begin(), sp64.end());
    int const nitems = static_cast<int>(items.size());
    // Marching tiles of a batch of 3D penalty-gauge problems.
    bool const march = std::all_of(probs.begin(), probs.end(), [](ProblemDesc const& q) {
        return q.dim == 3 && q.gauge == 0;
    });
    std::vector<Tile> tiles;
    if (march) {
        int const planes = march_planes(info, 4 * static_cast<int64_t>(multiprocessors()));
        for (int p = 0; p < np; ++p) {
            ProbInfo& pi = info[p];
            pi.first_tile = static_cast<int>(tiles.size());
            int idx = 0;
            for (int64_t k = 0; k < pi.nz; k += planes)
                for (int64_t j = 0; j < pi.ny; j += kMarchOwnRows)
                    for (int64_t i = 0; i < pi.nx; i += kMarchCols)
                        tiles.push_back({p, idx++, static_cast<int>(i), static_cast<int>(j), static_cast<int>(k),
                                         static_cast<int>(std::min(pi.nz, k + planes))});
            pi.ntiles = idx;
        }
    }
    int const ntiles = static_cast<int>(tiles.size());
    // Strips of a 2D batch.
    bool const flat = std::all_of(probs.begin(), probs.end(), [](ProblemDesc const& q) { return q.dim == 2; });
    int nstrip_ctas = 0;
    int const srows = flat ? strip_rows(info) : 0;
    std::vector<int> strip_part(np, 0);   // first strip CTA of each problem
    if (flat)
        for (int p = 0; p < np; ++p) {
            strip_part[p] = nstrip_ctas;
            nstrip_ctas += strips_of(info[p].nx, info[p].ny, srows).ctas;
        }
    int const nparts = std::max(std::max(nitems, ntiles), nstrip_ctas);
    // 2D problems that fit on chip are solved there; the others by the kernels
    // per iteration.
    std::vector<ResidentWave> const waves = flat ? plan_resident<T>(probs, chip_blocks(limits)) : std::vector<ResidentWave> {};
    size_t nres = 0;
    std::vector<char> resident(np, 0);
    for (ResidentWave const& w : waves) {
        nres += w.ctas.size();
        for (int p : w.probs) resident[p] = 1;
    }
    int const nvec = 8;  // x r z p q dinv nu p2 in precision T
    size_t const vec_bytes = ((total_rows * sizeof(T) + 255) / 256) * 256;
    size_t const d_bytes = ((total_rows * sizeof(double) + 255) / 256) * 256;
    size_t const ndouble_vecs = 3;  // nu64, r64, x64
    // Flexible CG ring: m stored directions and their images; m = 1 reuses p and q.
    int const fdirs = learned != nullptr ? (set.flexible_directions > 0 ? set.flexible_directions : 8) : 1;
    if (fdirs > kMaxDirs) return fail(SIL_ERR_INVALID, "flexible_directions exceeds 16");
    int const nhist = fdirs > 1 ? 2 * fdirs : 0;
    size_t bytes = (nvec + nhist) * vec_bytes + ndouble_vecs * d_bytes;
    // divergence-gauge coefficient tables (8 doubles + 8 floats per node)
    std::vector<size_t> gauge_off(np, 0);
    bool const any_gauge = std::any_of(probs.begin(), probs.end(), [](ProblemDesc const& q) {
        return q.dim == 3 && q.gauge != 0;
    });
    // the divergence-gauge variants only where a problem needs them
    auto const residual64 = any_gauge ? residual64_kernel<true> : residual64_kernel<false>;
    size_t gauge_bytes = 0;
    for (int p = 0; p < np; ++p) {
        if (probs[p].dim != 3 || probs[p].gauge == 0) continue;
        gauge_off[p] = gauge_bytes;
        gauge_bytes += ((static_cast<size_t>(info[p].nodes) * 8 * (sizeof(double) + sizeof(float)) + 255) / 256) * 256;
    }
    bytes += gauge_bytes + 256;
    bytes += sizeof(Item) * nitems + sizeof(ProbInfo) * np + sizeof(Vecs<T>) * np + sizeof(Scalars) * np
             + 3 * sizeof(double) * nparts + kMaxDirs * sizeof(double) * nitems + 7 * sizeof(void*) * np
             + sp64.size() * (sizeof(double) + sizeof(float)) + sizeof(int) * np + sizeof(int) * nitems
             + (sizeof(Tile) + sizeof(int)) * ntiles + sizeof(Work<T>) * nitems
             + sizeof(StripWork<T>) * nstrip_ctas
             + (sizeof(ResidentCta) + 2 * kMailSets * sizeof(unsigned long long)) * nres + 30 * 256;
    SolveBuffer buf;
    SIL_CUDA_CHECK(buf.take(bytes, stream));
    char* base = static_cast<char*>(buf.ptr);
    auto take = [&](size_t b) {
        char* r = base;
        base += (b + 255) / 256 * 256;
        return r;
    };
    T* vec_base[nvec];
    for (int k = 0; k < nvec; ++k) vec_base[k] = reinterpret_cast<T*>(take(vec_bytes));
    T* hist_base = nhist > 0 ? reinterpret_cast<T*>(take(nhist * vec_bytes)) : nullptr;
    int64_t const hstride = static_cast<int64_t>(vec_bytes / sizeof(T));
    double* nu64_base = reinterpret_cast<double*>(take(d_bytes));
    double* r64_base = reinterpret_cast<double*>(take(d_bytes));
    double* x64_base = reinterpret_cast<double*>(take(d_bytes));
    Item* d_items = reinterpret_cast<Item*>(take(sizeof(Item) * nitems));
    ProbInfo* d_info = reinterpret_cast<ProbInfo*>(take(sizeof(ProbInfo) * np));
    Vecs<T>* d_vecs = reinterpret_cast<Vecs<T>*>(take(sizeof(Vecs<T>) * np));
    Scalars* d_sc = reinterpret_cast<Scalars*>(take(sizeof(Scalars) * np));
    double* part_a = reinterpret_cast<double*>(take(sizeof(double) * nparts));
    double* part_b = reinterpret_cast<double*>(take(sizeof(double) * nparts));
    double* part_c = reinterpret_cast<double*>(take(sizeof(double) * nparts));
    double* part_h = reinterpret_cast<double*>(take(sizeof(double) * kMaxDirs * nitems));
    int* d_active = reinterpret_cast<int*>(take(sizeof(int) * np));
    int* d_act = reinterpret_cast<int*>(take(sizeof(int) * nitems));
    Work<T>* d_work = reinterpret_cast<Work<T>*>(take(sizeof(Work<T>) * nitems));
    ResidentCta* d_res = reinterpret_cast<ResidentCta*>(take(sizeof(ResidentCta) * nres));
    auto* d_mail = reinterpret_cast<unsigned long long*>(take(2 * kMailSets * sizeof(unsigned long long) * nres));
    StripWork<T>* d_strips = reinterpret_cast<StripWork<T>*>(take(sizeof(StripWork<T>) * nstrip_ctas));
    Tile* d_tiles = reinterpret_cast<Tile*>(take(sizeof(Tile) * ntiles));
    int* d_tact = reinterpret_cast<int*>(take(sizeof(int) * ntiles));
    char* gauge_base = gauge_bytes > 0 ? take(gauge_bytes) : nullptr;
    double const** d_mu = reinterpret_cast<double const**>(take(sizeof(void*) * np));
    double const** d_rhs = reinterpret_cast<double const**>(take(sizeof(void*) * np));
    double** d_nu64 = reinterpret_cast<double**>(take(sizeof(void*) * np));
    double** d_x64 = reinterpret_cast<double**>(take(sizeof(void*) * np));
    double** d_r64 = reinterpret_cast<double**>(take(sizeof(void*) * np));
    double** d_sol = reinterpret_cast<double**>(take(sizeof(void*) * np));
    double** d_scratch = reinterpret_cast<double**>(take(sizeof(void*) * np));
    double* d_sp64 = reinterpret_cast<double*>(take(sizeof(double) * sp64.size()));
    float* d_sp32 = reinterpret_cast<float*>(take(sizeof(float) * sp32.size()));
    for (int p = 0; p < np; ++p) {
        if (sp_off[p] < 0) continue;
        int64_t const len[3] = {info[p].nx, info[p].ny, info[p].nz};
        int64_t o = sp_off[p];
        for (int a = 0; a < 3; ++a) {
            info[p].ls64[a] = d_sp64 + o;
            info[p].ls32[a] = d_sp32 + o;
            o += len[a];
        }
        for (int a = 0; a < 3; ++a) {
            info[p].ils64[a] = d_sp64 + o;
            info[p].ils32[a] = d_sp32 + o;
            o += len[a];
        }
    }
    if (!sp64.empty()) {
        SIL_CUDA_CHECK(cudaMemcpyAsync(d_sp64, sp64.data(), sizeof(double) * sp64.size(), cudaMemcpyHostToDevice, stream));
        SIL_CUDA_CHECK(cudaMemcpyAsync(d_sp32, sp32.data(), sizeof(float) * sp32.size(), cudaMemcpyHostToDevice, stream));
    }
    // Divergence gauge tables, with the problem's slices of r64 / x64 as
    // probe scratch (both are rewritten before the solve reads them).
    {
        int64_t goff = 0;
        for (int p = 0; p < np; ++p) {
            if (probs[p].dim == 3 && probs[p].gauge != 0) {
                double* gd = reinterpret_cast<double*>(gauge_base + gauge_off[p]);
                float* g32 = reinterpret_cast<float*>(gd + 8 * info[p].nodes);
                info[p].gauge = 1;
                info[p].gd64 = gd;
                info[p].gd32 = g32;
                sil_status const gs = build_divergence_gauge(probs[p], info[p], gd, g32, r64_base + goff,
                                                             x64_base + goff, stream);
                if (gs != SIL_OK) return gs;
            }
            goff += info[p].n;
        }
    }

    std::vector<Vecs<T>> vecs(np);
    std::vector<double const*> mu(np), rhs(np);
    std::vector<double*> nu64(np), x64(np), r64(np);
    int64_t off = 0;
    for (int p = 0; p < np; ++p) {
        vecs[p] = {vec_base[0] + off, vec_base[1] + off, vec_base[2] + off, vec_base[3] + off,
                   vec_base[4] + off, vec_base[5] + off, vec_base[6] + off,
                   nhist > 0 ? hist_base + off : vec_base[3] + off,
                   nhist > 0 ? hist_base + fdirs * hstride + off : vec_base[4] + off, vec_base[7] + off};
        mu[p] = probs[p].node_mu;
        rhs[p] = probs[p].rhs;
        nu64[p] = nu64_base + off;
        x64[p] = x64_base + off;
        r64[p] = r64_base + off;
        off += info[p].n;
    }
    SIL_CUDA_CHECK(cudaMemcpyAsync(d_items, items.data(), sizeof(Item) * nitems, cudaMemcpyHostToDevice, stream));
    if (ntiles > 0)
        SIL_CUDA_CHECK(cudaMemcpyAsync(d_tiles, tiles.data(), sizeof(Tile) * ntiles, cudaMemcpyHostToDevice, stream));
    SIL_CUDA_CHECK(cudaMemcpyAsync(d_info, info.data(), sizeof(ProbInfo) * np, cudaMemcpyHostToDevice, stream));
    SIL_CUDA_CHECK(cudaMemcpyAsync(d_vecs, vecs.data(), sizeof(Vecs<T>) * np, cudaMemcpyHostToDevice, stream));
    SIL_CUDA_CHECK(cudaMemcpyAsync(d_mu, mu.data(), sizeof(void*) * np, cudaMemcpyHostToDevice, stream));
    SIL_CUDA_CHECK(cudaMemcpyAsync(d_rhs, rhs.data(), sizeof(void*) * np, cudaMemcpyHostToDevice, stream));
    SIL_CUDA_CHECK(cudaMemcpyAsync(d_nu64, nu64.data(), sizeof(void*) * np, cudaMemcpyHostToDevice, stream));
    SIL_CUDA_CHECK(cudaMemcpyAsync(d_x64, x64.data(), sizeof(void*) * np, cudaMemcpyHostToDevice, stream));
    SIL_CUDA_CHECK(cudaMemcpyAsync(d_r64, r64.data(), sizeof(void*) * np, cudaMemcpyHostToDevice, stream));
    std::vector<double*> sol(np), scratch(np);
    for (int p = 0; p < np; ++p) {
        sol[p] = probs[p].solution;
        scratch[p] = r64[p];  // FP64 scratch for the final true residual
    }
    SIL_CUDA_CHECK(cudaMemcpyAsync(d_sol, sol.data(), sizeof(void*) * np, cudaMemcpyHostToDevice, stream));
    SIL_CUDA_CHECK(cudaMemcpyAsync(d_scratch, scratch.data(), sizeof(void*) * np, cudaMemcpyHostToDevice, stream));
    SIL_CUDA_CHECK(cudaMemsetAsync(d_sc, 0, sizeof(Scalars) * np, stream));

    setup_kernel<T><<<nitems, kThreads, 0, stream>>>(d_items, d_info, d_mu, d_nu64, d_vecs);
    SIL_CUDA_CHECK(cudaGetLastError());

    double const tol = set.relative_tolerance > 0 ? set.relative_tolerance : 1e-10;
    int const max_iter = set.max_iterations > 0 ? set.max_iterations : 100000;
    int const chunk = 32;
    std::vector<Scalars> hs(np);

    // Items of the problems not yet converged (the CG kernels skip problems
    // whose inner solve has stopped); a chunk of iterations over them is
    // captured as a CUDA graph, captured again once the list has shrunk by a
    // tenth (a longer list is still correct: its finished problems return at
    // once).
    std::vector<int> open_host;
    open_host.reserve(nitems);
    int captured_n = -1;
    std::vector<int> open_tiles;
    std::vector<Work<T>> work;
    std::vector<StripWork<T>> swork;
    int captured_tiles = 0, captured_strips = 0;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    auto build_open = [&]() {
        open_host.clear();
        for (int i = 0; i < nitems; ++i)
            if (!hs[items[i].prob].outer_done && !resident[items[i].prob]) open_host.push_back(i);
        open_tiles.clear();
        for (int i = 0; i < ntiles; ++i)
            if (!hs[tiles[i].prob].outer_done) open_tiles.push_back(i);
    };
    // The strips of the open problems of a 2D batch.
    auto build_strips = [&](std::vector<char> const& open) {
        swork.clear();
        for (int p = 0; flat && p < np; ++p) {
            if (!open[p]) continue;
            ProbInfo const& pi = info[p];
            Vecs<T> const& v = vecs[p];
            Strips const st = strips_of(pi.nx, pi.ny, srows);
            for (int k = 0; k < st.ctas; ++k)
                swork.push_back({v.x, v.z, v.p, v.p2, v.q, v.nu, d_sc + p, part_a + strip_part[p], part_b + pi.first_item,
                                 part_c + pi.first_item, static_cast<int>(pi.nx), static_cast<int>(pi.ny), st.strips,
                                 st.rows, st.count, k * kStripWarps, k, p, pi.nitems, pi.max_iters});
        }
    };
    auto capture_chunk = [&]() -> sil_status {
        if (exec != nullptr) cudaGraphExecDestroy(exec);
        if (graph != nullptr) cudaGraphDestroy(graph);
        exec = nullptr;
        graph = nullptr;
        int const n = static_cast<int>(open_host.size()), nt = static_cast<int>(open_tiles.size());
        SIL_CUDA_CHECK(cudaMemcpyAsync(d_act, open_host.data(), sizeof(int) * n, cudaMemcpyHostToDevice, stream));
        work.clear();
        for (int i : open_host) {
            Item const& it = items[i];
            ProbInfo const& pi = info[it.prob];
            Vecs<T> const& v = vecs[it.prob];
            work.push_back({v.x, v.r, v.z, v.p, v.q, v.dinv, d_sc + it.prob,
                            part_a + (march ? pi.first_tile : (flat ? strip_part[it.prob] : pi.first_item)),
                            part_b + pi.first_item, part_c + pi.first_item, static_cast<int>(it.begin),
                            static_cast<int>(it.end), it.index, pi.nitems,
                            march ? pi.ntiles : (flat ? strips_of(pi.nx, pi.ny, srows).ctas : pi.nitems), pi.max_iters});
        }
        std::vector<char> open(np, 0);
        for (int i : open_host) open[items[i].prob] = 1;
        build_strips(open);
        int const ns = static_cast<int>(swork.size());
        if (ns > 0)
            SIL_CUDA_CHECK(cudaMemcpyAsync(d_strips, swork.data(), sizeof(StripWork<T>) * ns, cudaMemcpyHostToDevice,
                                           stream));
        SIL_CUDA_CHECK(cudaMemcpyAsync(d_work, work.data(), sizeof(Work<T>) * n, cudaMemcpyHostToDevice, stream));
        if (nt > 0)
            SIL_CUDA_CHECK(cudaMemcpyAsync(d_tact, open_tiles.data(), sizeof(int) * nt, cudaMemcpyHostToDevice, stream));
        cudaStream_t cs;
        SIL_CUDA_CHECK(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
        cudaError_t err = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
        for (int c = 0; c < chunk && err == cudaSuccess; ++c) {
            if (march) {
                cg_direction3_kernel<T><<<n, kThreads, 0, cs>>>(d_work, c);
                cg_march_kernel<T><<<nt, kMarchThreads, 0, cs>>>(d_tiles, d_tact, d_info, d_vecs, d_sc, part_a, c);
            } else if (any_gauge) {
                cg_direction3_kernel<T><<<n, kThreads, 0, cs>>>(d_work, c);
                cg_apply3_kernel<T><<<n, kThreads, 0, cs>>>(d_items, d_act, d_info, d_vecs, d_sc, part_a, c);
            } else {
                cg_direction2_kernel<T><<<ns, kThreads, 0, cs>>>(d_strips, c);
            }
            if (flat) cg_update_kernel<T, true><<<n, kThreads, 0, cs>>>(d_work, c);
            else cg_update_kernel<T, false><<<n, kThreads, 0, cs>>>(d_work, c);
        }
        if (flat) cg_close_kernel<T, false><<<n, kThreads, 0, cs>>>(d_work, chunk);
        else cg_close_kernel<T, true><<<n, kThreads, 0, cs>>>(d_work, chunk);
        cudaError_t const err2 = cudaStreamEndCapture(cs, &graph);
        if (err == cudaSuccess) err = err2;
        if (err == cudaSuccess) err = cudaGraphInstantiate(&exec, graph, 0);
        cudaStreamDestroy(cs);
        if (err != cudaSuccess) return cuda_fail(err, "solver graph capture");
        captured_n = n;
        captured_tiles = nt;
        captured_strips = ns;
        return SIL_OK;
    };
    auto read_scalars = [&]() -> sil_status {
        SIL_CUDA_CHECK(cudaMemcpyAsync(hs.data(), d_sc, sizeof(Scalars) * np, cudaMemcpyDeviceToHost, stream));
        SIL_CUDA_CHECK(cudaStreamSynchronize(stream));
        return SIL_OK;
    };

    // Iterative refinement on the FP64 residual with reliable updates: after
    // every chunk of CG iterations in precision T, x64 += ||r|| x, the FP64
    // true residual r = b - A x64 replaces the recurrence's residual, and CG
    // continues with its previous search direction (residual replacement,
    // not a restart), so the Krylov space survives and the recurrence never
    // drifts far from the true residual.  A problem stops iterating once its
    // recurrence reaches half the outer tolerance and converges once the
    // FP64 residual does.  With T = float the chunks run at half the bytes
    // of FP64 and converge at nearly the FP64 rate.
    sil_status st = SIL_OK;
    int refinements = 0;
    SIL_CUDA_CHECK(cudaMemsetAsync(x64_base, 0, d_bytes, stream));

    // Refinement passes whose inner solve is the flexible CG preconditioned by
    // the learned network, until every problem has converged or been handed to
    // the plain solver (stall or budget).
    auto learned_stage = [&](nn::Net* net, int* total_out, int* refinements_out) -> sil_status {
        if constexpr (!std::is_same_v<T, float>) {
            return fail(SIL_ERR_UNSUPPORTED, "learned solve runs in FP32");
        } else {
            std::vector<nn::Sample> samples(np);
            int64_t o = 0;
            for (int p = 0; p < np; ++p) {
                if (info[p].dim != 2) return fail(SIL_ERR_UNSUPPORTED, "learned solve: 2D problems only");
                samples[p] = {static_cast<int32_t>(info[p].nx), static_cast<int32_t>(info[p].ny), o};
                o += info[p].n;
            }
            nn::Workspace* ws = nullptr;
            sil_status lst = net->prepare(samples, stream, &ws);
            if (lst != SIL_OK) return lst;
            // nu is fixed for the whole solve: the network's log(nu) input is formed once
            lst = net->set_static_nu(ws, vec_base[6], stream);
            if (lst != SIL_OK) return lst;
            float const* nuf = vec_base[6];
            float const* dv = vec_base[5];
            float* rv = vec_base[1];
            float* zv = vec_base[2];
            int const window = set.stall_window > 0 ? set.stall_window : 200;
            double const ltol = set.inner_tolerance > 0 ? set.inner_tolerance : 1e-5;
            int const lmax = set.inner_iterations > 0 ? set.inner_iterations : 4000;
            int const lchunk = 8;
            int ln = 0;  // items the flexible CG's kernels visit (listed in d_act)
            // z -> A-orthogonal direction in the next ring slot.
            auto new_direction = [&](cudaStream_t cs) {
                if (fdirs <= 1) {
                    fcg_orth_kernel<T, 1><<<ln, kThreads, 0, cs>>>(d_items, d_act, d_info, d_vecs, d_sc, part_h, hstride, fdirs,
                                                                    nitems);
                    fcg_direction_kernel<T, 1><<<ln, kThreads, 0, cs>>>(d_items, d_act, d_vecs, d_sc, hstride, fdirs);
                } else if (fdirs <= 4) {
                    fcg_orth_kernel<T, 4><<<ln, kThreads, 0, cs>>>(d_items, d_act, d_info, d_vecs, d_sc, part_h, hstride, fdirs,
                                                                    nitems);
                    fcg_direction_kernel<T, 4><<<ln, kThreads, 0, cs>>>(d_items, d_act, d_vecs, d_sc, hstride, fdirs);
                } else if (fdirs <= 8) {
                    fcg_orth_kernel<T, 8><<<ln, kThreads, 0, cs>>>(d_items, d_act, d_info, d_vecs, d_sc, part_h, hstride, fdirs,
                                                                    nitems);
                    fcg_direction_kernel<T, 8><<<ln, kThreads, 0, cs>>>(d_items, d_act, d_vecs, d_sc, hstride, fdirs);
                } else {
                    fcg_orth_kernel<T, 16><<<ln, kThreads, 0, cs>>>(d_items, d_act, d_info, d_vecs, d_sc, part_h, hstride, fdirs,
                                                                    nitems);
                    fcg_direction_kernel<T, 16><<<ln, kThreads, 0, cs>>>(d_items, d_act, d_vecs, d_sc, hstride, fdirs);
                }
            };
            // The flexible CG's kernels visit the items of the problems still
            // iterating (`ln` of them, listed in d_act); the chunk graph is
            // captured again once that list has shrunk by a tenth.
            cudaGraph_t lgraph = nullptr;
            cudaGraphExec_t lexec = nullptr;
            std::vector<int> lopen;
            lopen.reserve(nitems);
            auto build_lopen = [&]() {
                lopen.clear();
                for (int i = 0; i < nitems; ++i) {
                    Scalars const& q = hs[items[i].prob];
                    if (!q.outer_done && !q.fallback && !q.done) lopen.push_back(i);
                }
            };
            auto capture_learned = [&]() -> sil_status {
                if (lexec != nullptr) cudaGraphExecDestroy(lexec);
                if (lgraph != nullptr) cudaGraphDestroy(lgraph);
                lexec = nullptr;
                lgraph = nullptr;
                ln = static_cast<int>(lopen.size());
                std::vector<char> open(np, 0);
                for (int i : lopen) open[items[i].prob] = 1;
                build_strips(open);
                int const lstrips = static_cast<int>(swork.size());
                SIL_CUDA_CHECK(cudaMemcpyAsync(d_strips, swork.data(), sizeof(StripWork<T>) * lstrips,
                                               cudaMemcpyHostToDevice, stream));
                SIL_CUDA_CHECK(cudaMemcpyAsync(d_act, lopen.data(), sizeof(int) * ln, cudaMemcpyHostToDevice, stream));
                cudaStream_t cs;
                SIL_CUDA_CHECK(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
                sil_status cst = SIL_OK;
                cudaError_t err = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
                for (int c = 0; c < lchunk && err == cudaSuccess && cst == SIL_OK; ++c) {
                    fcg_apply_kernel<T><<<lstrips, kThreads, 0, cs>>>(d_strips, d_vecs, hstride, fdirs, part_b - part_a);
                    fcg_update_kernel<T><<<ln, kThreads, 0, cs>>>(d_items, d_act, d_info, d_vecs, d_sc, part_c, window,
                                                                  hstride, fdirs, d_active);
                    cst = net->forward(ws, nuf, dv, rv, zv, cs, d_active);
                    new_direction(cs);
                }
                cudaError_t const err2 = cudaStreamEndCapture(cs, &lgraph);
                if (err == cudaSuccess) err = err2;
                if (err == cudaSuccess && cst == SIL_OK) err = cudaGraphInstantiate(&lexec, lgraph, 0);
                cudaStreamDestroy(cs);
                if (cst != SIL_OK) return cst;
                if (err != cudaSuccess) return cuda_fail(err, "learned solver graph capture");
                return SIL_OK;
            };
            int tot = 0;
            while (lst == SIL_OK && tot < max_iter) {
                residual64<<<nitems, kThreads, 0, stream>>>(d_items, nullptr, d_info, d_nu64, d_rhs, d_x64, d_r64,
                                                                   d_sc, part_a, tol * tol, ltol * ltol, 1);
                SIL_CUDA_CHECK(cudaMemcpyAsync(hs.data(), d_sc, sizeof(Scalars) * np, cudaMemcpyDeviceToHost, stream));
                SIL_CUDA_CHECK(cudaStreamSynchronize(stream));
                bool active = false;
                for (int p = 0; p < np; ++p) active = active || (!hs[p].outer_done && !hs[p].fallback);
                if (!active) break;
                fcg_init_kernel<T><<<nitems, kThreads, 0, stream>>>(d_items, nullptr, d_info, d_vecs, d_r64, d_sc, part_a,
                                                                    *refinements_out == 0 ? 1 : 0);
                // every problem not converged and not handed over iterates after the init
                for (int p = 0; p < np; ++p) hs[p].done = 0;
                build_lopen();
                lst = capture_learned();
                if (lst != SIL_OK) break;
                fcg_active_kernel<<<(np + 63) / 64, 64, 0, stream>>>(d_sc, np, d_active);
                lst = net->forward(ws, nuf, dv, rv, zv, stream, d_active);
                if (lst != SIL_OK) break;
                new_direction(stream);
                SIL_CUDA_CHECK(cudaGetLastError());
                int const budget = std::min(lmax, max_iter - tot);
                int spent = 0;
                while (spent < budget) {
                    SIL_CUDA_CHECK(cudaGraphLaunch(lexec, stream));
                    spent += lchunk;
                    SIL_CUDA_CHECK(cudaMemcpyAsync(hs.data(), d_sc, sizeof(Scalars) * np, cudaMemcpyDeviceToHost, stream));
                    SIL_CUDA_CHECK(cudaStreamSynchronize(stream));
                    build_lopen();
                    if (lopen.empty()) break;
                    if (10 * static_cast<int>(lopen.size()) < 9 * ln) {
                        lst = capture_learned();
                        if (lst != SIL_OK) break;
                    }
                }
                if (lst != SIL_OK) break;
                tot += spent;
                // A problem still unconverged after a full inner budget goes to the plain solver.
                bool flagged = false;
                for (int p = 0; p < np; ++p) {
                    if (!hs[p].outer_done && !hs[p].fallback && !hs[p].done) {
                        hs[p].fallback = 1;
                        flagged = true;
                    }
                }
                refine_kernel<T><<<nitems, kThreads, 0, stream>>>(d_items, nullptr, d_vecs, d_x64, d_sc);
                if (flagged) {
                    SIL_CUDA_CHECK(cudaMemcpyAsync(d_sc, hs.data(), sizeof(Scalars) * np, cudaMemcpyHostToDevice, stream));
                }
                ++*refinements_out;
            }
            if (lexec != nullptr) cudaGraphExecDestroy(lexec);
            if (lgraph != nullptr) cudaGraphDestroy(lgraph);
            net->set_static_nu(ws, nullptr, stream);
            *total_out = tot;
            return lst;
        }
    };
    // bb = ||b||^2 via an init pass from the right-hand side.
    cg_init_kernel<T><<<nitems, kThreads, 0, stream>>>(d_items, d_info, d_vecs, d_rhs, nullptr, d_sc, part_a, part_b,
                                                       false);
    int total = 0, resident_cycles = 0;
    if constexpr (std::is_same_v<T, float>) {
        if (learned != nullptr && st == SIL_OK) st = learned_stage(learned, &total, &refinements);
    }
    // The resident problems, wave after wave.
    if (st == SIL_OK && !waves.empty()) {
        std::vector<ResidentCta> all;
        for (ResidentWave const& w : waves) all.insert(all.end(), w.ctas.begin(), w.ctas.end());
        SIL_CUDA_CHECK(cudaMemcpyAsync(d_res, all.data(), sizeof(ResidentCta) * all.size(), cudaMemcpyHostToDevice, stream));
        std::vector<unsigned long long> const empty(2 * kMailSets * nres, kNoMail);
        SIL_CUDA_CHECK(cudaMemcpyAsync(d_mail, empty.data(), sizeof(unsigned long long) * empty.size(),
                                       cudaMemcpyHostToDevice, stream));
        size_t at = 0;
        for (ResidentWave const& w : waves) {
            void const* const kernel = resident_kernel<T>(w.per_thread);
            ResidentCta const* ctas = d_res + at;
            double tol2 = tol * tol;
            int budget = max_iter, spent = total, steps = chunk;
            int polls = limits.wait_polls < 0 ? kResPollLimit : limits.wait_polls;
            void* args[] = {&ctas, &d_vecs, &d_nu64, &d_rhs, &d_x64, &d_r64, &d_sc, &d_mail, &tol2, &budget, &spent, &steps, &polls};
            cudaError_t refused = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                       static_cast<int>(kResSmemMost));
            if (refused == cudaSuccess)
                refused = cudaLaunchCooperativeKernel(kernel, dim3(static_cast<unsigned>(w.ctas.size())),
                                                      dim3(kResThreads), args, w.smem, stream);
            if (refused != cudaSuccess) {
                // not run: the kernels per iteration take its problems (an error
                // that outlasts the launch comes back from the next call)
                cudaGetLastError();
                for (int p : w.probs) resident[p] = 0;
                limits.handed_over += static_cast<int>(w.probs.size());
            }
            at += w.ctas.size();
        }
        st = read_scalars();
        if (st != SIL_OK) return st;
        int cycles = 0;
        for (int p = 0; p < np; ++p) {
            cycles = std::max(cycles, hs[p].cycles);
            if (!resident[p] || !hs[p].timeout || hs[p].outer_done) continue;
            // A wait ran out (the group's blocks were kept from running for
            // seconds): the kernels per iteration go on from its x64, of whose
            // rows some may hold a correction that the others still lack.
            resident[p] = 0;
            ++limits.handed_over;
        }
        resident_cycles = cycles;
    }
    limits.solved = static_cast<int>(std::count(resident.begin(), resident.end(), 1));
    // Cycle: FP64 residual (outer check) -> residual replacement -> a chunk
    // of iterations -> x64 += ||r|| x; the host reads the problems' state
    // once per cycle.
    auto const residual_open = any_gauge ? residual64_kernel<true> : residual64_kernel<false>;
    int const before = refinements;
    build_open();
    if (st == SIL_OK && !open_host.empty()) st = capture_chunk();
    bool fresh = true;
    while (st == SIL_OK && !open_host.empty()) {
        int const n = captured_n;
        if (march)
            residual64_march_kernel<<<captured_tiles, kMarchThreads, 0, stream>>>(
                    d_tiles, d_tact, d_info, d_nu64, d_rhs, d_x64, d_r64, d_sc, part_a, tol * tol, 0.0, 1);
        else if (flat)
            residual64_strip_kernel<T><<<captured_strips, kThreads, 0, stream>>>(d_strips, d_nu64, d_rhs, d_x64, d_r64,
                                                                                 tol * tol, 0.0, 1);
        else
            residual_open<<<n, kThreads, 0, stream>>>(d_items, d_act, d_info, d_nu64, d_rhs, d_x64, d_r64, d_sc, part_a,
                                                      tol * tol, 0.0, 1);
        st = read_scalars();
        if (st != SIL_OK) break;
        build_open();
        if (open_host.empty() || total >= max_iter) break;
        if (10 * static_cast<int>(open_host.size()) < 9 * captured_n) {
            st = capture_chunk();
            if (st != SIL_OK) break;
        }
        cg_replace_kernel<T><<<captured_n, kThreads, 0, stream>>>(d_items, d_act, d_info, d_vecs, d_r64, d_sc,
                                                                  part_a, part_b, fresh ? 1 : 0);
        SIL_CUDA_CHECK(cudaGetLastError());
        fresh = false;
        SIL_CUDA_CHECK(cudaGraphLaunch(exec, stream));
        total += chunk;
        refine_kernel<T><<<captured_n, kThreads, 0, stream>>>(d_items, d_act, d_vecs, d_x64, d_sc);
        ++refinements;
    }
    refinements = std::max(refinements, before + resident_cycles);
    if (exec != nullptr) cudaGraphExecDestroy(exec);
    if (graph != nullptr) cudaGraphDestroy(graph);
    if (st == SIL_OK) copy_kernel<<<nitems, kThreads, 0, stream>>>(d_items, d_x64, d_sol, d_sc);
    if (st != SIL_OK) return st;

    // FP64 true residual ||b - A x|| of the returned solution for every problem.
    std::vector<Scalars> hs2(np);
    SIL_CUDA_CHECK(cudaMemcpyAsync(hs2.data(), d_sc, sizeof(Scalars) * np, cudaMemcpyDeviceToHost, stream));
    SIL_CUDA_CHECK(cudaStreamSynchronize(stream));
    for (int p = 0; p < np; ++p) {
        hs2[p].outer_done = 0;
        hs2[p].counter_a = hs2[p].counter_c = 0;
    }
    SIL_CUDA_CHECK(cudaMemcpyAsync(d_sc, hs2.data(), sizeof(Scalars) * np, cudaMemcpyHostToDevice, stream));
    residual64<<<nitems, kThreads, 0, stream>>>(d_items, nullptr, d_info, d_nu64, d_rhs, d_sol, d_scratch, d_sc,
                                                       part_a, tol * tol, 0.0, 0);
    SIL_CUDA_CHECK(cudaGetLastError());
    SIL_CUDA_CHECK(cudaMemcpyAsync(hs.data(), d_sc, sizeof(Scalars) * np, cudaMemcpyDeviceToHost, stream));
    SIL_CUDA_CHECK(cudaStreamSynchronize(stream));
    sil_status overall = SIL_OK;
    for (int p = 0; p < np; ++p) {
        sil_solve_diagnostics& d = diag[p];
        d.iterations = hs[p].total_iters;
        d.refinements = refinements;
        d.initial_residual_l2 = std::sqrt(hs[p].bb);
        d.final_residual_l2 = std::sqrt(hs[p].rr);
        d.final_relative_residual = hs[p].bb > 0 ? std::sqrt(hs[p].rr / hs[p].bb) : 0.0;
        d.converged = d.final_relative_residual <= tol && !hs[p].nonfinite;
        d.status = hs[p].nonfinite ? SIL_ERR_NONFINITE : SIL_OK;
        d.learned_iterations = hs[p].learned_iters;
        d.fallback = hs[p].fallback;
        if (hs[p].nonfinite) overall = SIL_ERR_NONFINITE;
    }
    if (overall != SIL_OK) set_error("a problem of the batch met a non-finite value");
    return overall;
}

// Work-item size of the batched CG kernels, picked by timing.  The first
// batch of at least 4 M rows solved in a precision (2D and 3D batches apart)
// runs a 96-iteration solve with items of 2,048, 4,096 and 8,192 rows and
// keeps the fastest for such batches of the process (the tuning solves write the
// caller's solution buffers, which the real solve overwrites).  Smaller
// batches take the rows that make one wave, at most 4,096.
// SIMILIE_B200_ITEM_ROWS=<rows> forces a size; SIMILIE_B200_AUTOTUNE=0 keeps
// the default.  (Whatever the size, a problem has at most one wave of items:
// item_step.)
constexpr int kItemCandidates[3] = {2048, 4096, 8192};
std::mutex g_item_mutex;
int g_item_rows_tuned[4] = {0, 0, 0, 0};  // [precision FP64 / FP32][first problem 2D / 3D]

template <class T>
sil_status choose_item_rows(std::vector<ProblemDesc> const& probs, sil_solve_settings const& set, cudaStream_t stream,
                            sil_chip_limits const& limits, int* rows)
{
    int64_t total = 0;
    for (ProblemDesc const& q : probs) total += (q.dim == 3 ? 3 : 1) * q.nx * q.ny * (q.dim == 3 ? q.nz : 1);
    // small batches: one wave of four CTAs per multiprocessor (fewer than two
    // rows a thread cost more in partials than they gain)
    int64_t const wave = 4 * static_cast<int64_t>(multiprocessors());
    int64_t const spread = ((total + wave - 1) / wave + kThreads - 1) / kThreads * kThreads;
    *rows = static_cast<int>(std::max<int64_t>(2 * kThreads, std::min<int64_t>(kItemNodes, spread)));
    if (char const* e = std::getenv("SIMILIE_B200_ITEM_ROWS")) {
        int const v = std::atoi(e);
        if (v >= kThreads && v % kThreads == 0 && v <= 64 * kThreads) {
            *rows = v;
            return SIL_OK;
        }
    }
    if (total < (int64_t(1) << 22)) return SIL_OK;
    int const blocks = chip_blocks(limits);
    if (std::all_of(probs.begin(), probs.end(), [&](ProblemDesc const& q) { return resident_ctas<T>(q, blocks) > 0; }))
        return SIL_OK;   // solved on chip
    int const key = (sizeof(T) == 8 ? 0 : 2) + (probs.front().dim == 3 ? 1 : 0);
    {
        std::lock_guard<std::mutex> lock(g_item_mutex);
        if (g_item_rows_tuned[key] > 0) {
            *rows = g_item_rows_tuned[key];
            return SIL_OK;
        }
    }
    char const* at = std::getenv("SIMILIE_B200_AUTOTUNE");
    if (at != nullptr && at[0] == '0') return SIL_OK;
    sil_solve_settings probe = set;
    probe.max_iterations = 96;
    std::vector<sil_solve_diagnostics> scratch(probs.size());
    double best = 1e300;
    int best_rows = kItemNodes;
    for (int c : kItemCandidates) {
        auto const t0 = std::chrono::steady_clock::now();
        sil_chip_limits within = limits;
        sil_status const st = solve_batch_rows<T>(probs, probe, scratch.data(), stream, nullptr, within, c);
        if (st != SIL_OK) return st;
        double const sec = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
        if (sec < best) {
            best = sec;
            best_rows = c;
        }
    }
    std::lock_guard<std::mutex> lock(g_item_mutex);
    g_item_rows_tuned[key] = best_rows;
    *rows = best_rows;
    return SIL_OK;
}

template <class T>
sil_status solve_batch(std::vector<ProblemDesc> const& probs, sil_solve_settings const& set, sil_solve_diagnostics* diag,
                       cudaStream_t stream, sil_chip_limits& limits, nn::Net* learned = nullptr)
{
    int rows = kItemNodes;
    sil_status const st = choose_item_rows<T>(probs, set, stream, limits, &rows);
    if (st != SIL_OK) return st;
    return solve_batch_rows<T>(probs, set, diag, stream, learned, limits, rows);
}

} // namespace

} // namespace sil

using namespace sil;

extern "C" {

sil_status sil_mag2d_apply(sil_stream stream, int64_t nx, int64_t ny, const double* node_mu, const double* a, double* y)
{
    if (nx < 3 || ny < 3) return fail(SIL_ERR_INVALID, "sil_mag2d_apply: need at least 3x3 nodes");
    if (nx * ny >= (int64_t(1) << 31)) return fail(SIL_ERR_INVALID, "sil_mag2d_apply: fewer than 2^31 nodes supported");
    if (node_mu == nullptr || a == nullptr || y == nullptr) return fail(SIL_ERR_INVALID, "sil_mag2d_apply: NULL pointer");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    int64_t const n = nx * ny;
    DeviceBuffer nu;
    SIL_CUDA_CHECK(cudaMallocAsync(&nu.ptr, n * sizeof(double), s));
    int const blocks = static_cast<int>((n + 255) / 256);
    reciprocal_kernel<<<blocks, 256, 0, s>>>(node_mu, static_cast<double*>(nu.ptr), n);
    mag_apply_kernel<<<blocks, 256, 0, s>>>(static_cast<double*>(nu.ptr), a, y, nx, ny);
    SIL_CUDA_CHECK(cudaGetLastError());
    SIL_CUDA_CHECK(cudaFreeAsync(nu.ptr, s));
    nu.ptr = nullptr;
    return SIL_OK;
}

} // extern "C"

// ------------------------------------------------------------------ allocation-free apply

namespace sil {
namespace {

// Scratch of sil_mag2d_apply_noalloc: the reciprocal permeability 1/mu of
// every node.  A fixed array in the library's device image (16 MiB of
// doubles), so the entry point never allocates; every GPU that loads the
// library holds it until the process exits.
constexpr int64_t kNoAllocMaxNodes = int64_t(1) << 21;
static __device__ __align__(256) double g_noalloc_nu[kNoAllocMaxNodes];

constexpr int kNoAllocMaxDevices = 128;
std::mutex g_noalloc_mutex;
double* g_noalloc_ptr[kNoAllocMaxDevices] = {};

// Device address of the scratch array on the current device.  The host-side
// name g_noalloc_nu is only a stand-in for the symbol; its device address is
// looked up once per device, with that device current.
sil_status noalloc_scratch(double** out)
{
    int dev = 0;
    SIL_CUDA_CHECK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kNoAllocMaxDevices) return fail(SIL_ERR_UNSUPPORTED, "sil_mag2d_apply_noalloc: device index too large");
    std::lock_guard<std::mutex> lock(g_noalloc_mutex);
    if (g_noalloc_ptr[dev] == nullptr) {
        void* p = nullptr;
        cudaError_t const err = cudaGetSymbolAddress(&p, g_noalloc_nu);
        if (err != cudaSuccess) return cuda_fail(err, "sil_mag2d_apply_noalloc: cudaGetSymbolAddress");
        g_noalloc_ptr[dev] = static_cast<double*>(p);
    }
    *out = g_noalloc_ptr[dev];
    return SIL_OK;
}

} // namespace
} // namespace sil

extern "C" {

sil_status sil_mag2d_apply_noalloc(sil_stream stream, int64_t nx, int64_t ny, const double* node_mu, const double* a,
                                   double* y)
{
    if (nx < 3 || ny < 3) return fail(SIL_ERR_INVALID, "sil_mag2d_apply_noalloc: need at least 3x3 nodes");
    if (node_mu == nullptr || a == nullptr || y == nullptr)
        return fail(SIL_ERR_INVALID, "sil_mag2d_apply_noalloc: NULL pointer");
    if (nx > kNoAllocMaxNodes || ny > kNoAllocMaxNodes || nx * ny > kNoAllocMaxNodes)
        return fail(SIL_ERR_INVALID, "sil_mag2d_apply_noalloc: nx*ny = " + std::to_string(nx * ny)
                                             + " exceeds the fixed scratch of " + std::to_string(kNoAllocMaxNodes)
                                             + " nodes; use sil_mag2d_apply");
    double* nu = nullptr;
    sil_status const st = noalloc_scratch(&nu);
    if (st != SIL_OK) return st;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    int64_t const n = nx * ny;
    int const blocks = static_cast<int>((n + 255) / 256);
    // Every scratch entry the apply reads is written first, so nothing from a
    // previous call needs clearing.
    reciprocal_kernel<<<blocks, 256, 0, s>>>(node_mu, nu, n);
    mag_apply_kernel<<<blocks, 256, 0, s>>>(nu, a, y, nx, ny);
    SIL_CUDA_CHECK(cudaGetLastError());
    return SIL_OK;
}

sil_status sil_mag2d_solve_batch(const sil_mag2d_problem* problems, int nproblems, const sil_solve_settings* settings,
                                 sil_solve_diagnostics* diag, sil_stream stream)
{
    sil_chip_limits limits = {-1, -1, 0, 0};
    return sil_mag2d_solve_batch_within(&limits, problems, nproblems, settings, diag, stream);
}

sil_status sil_mag2d_solve_batch_within(sil_chip_limits* limits, const sil_mag2d_problem* problems, int nproblems,
                                        const sil_solve_settings* settings, sil_solve_diagnostics* diag,
                                        sil_stream stream)
{
    if (limits == nullptr || limits->blocks < -1 || limits->wait_polls < -1)
        return fail(SIL_ERR_INVALID, "sil_mag2d_solve_batch_within: NULL or bad limits");
    limits->solved = limits->handed_over = 0;
    if (problems == nullptr || settings == nullptr || diag == nullptr || nproblems < 1)
        return fail(SIL_ERR_INVALID, "sil_mag2d_solve_batch: NULL argument or empty batch");
    std::vector<ProblemDesc> descs(nproblems);
    for (int p = 0; p < nproblems; ++p) {
        sil_mag2d_problem const& q = problems[p];
        if (q.nx < 3 || q.ny < 3) return fail(SIL_ERR_INVALID, "sil_mag2d_solve_batch: each problem needs >= 3x3 nodes");
        if (q.nx * q.ny >= (int64_t(1) << 31))
            return fail(SIL_ERR_INVALID, "sil_mag2d_solve_batch: a problem must have fewer than 2^31 nodes");
        if (q.node_mu == nullptr || q.rhs == nullptr || q.solution == nullptr)
            return fail(SIL_ERR_INVALID, "sil_mag2d_solve_batch: NULL field pointer");
        descs[p] = {2, q.nx, q.ny, 1, 0.0, q.node_mu, q.rhs, q.solution, {nullptr, nullptr, nullptr}};
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    std::memset(diag, 0, sizeof(sil_solve_diagnostics) * nproblems);
    if (settings->solver == SIL_SOLVER_CG_F64) return solve_batch<double>(descs, *settings, diag, s, *limits);
    if (settings->solver == SIL_SOLVER_MIXED_IR) return solve_batch<float>(descs, *settings, diag, s, *limits);
    if (settings->solver == SIL_SOLVER_LEARNED) {
        if (settings->preconditioner == nullptr)
            return fail(SIL_ERR_INVALID, "sil_mag2d_solve_batch: the learned solver needs a preconditioner");
        if (nproblems > nn::kMaxImages)
            return fail(SIL_ERR_INVALID, "sil_mag2d_solve_batch: the learned solver takes at most 64 problems per call");
        return solve_batch<float>(descs, *settings, diag, s, *limits, &settings->preconditioner->net);
    }
    return fail(SIL_ERR_INVALID, "sil_mag2d_solve_batch: unknown solver kind");
}

} // extern "C"

// ------------------------------------------------------------------ 3D

namespace sil {
namespace {

sil_status check_mag3d(sil_mag3d_problem const& q, char const* who, bool need_fields)
{
    if (q.nx < 3 || q.ny < 3 || q.nz < 3) return fail(SIL_ERR_INVALID, std::string(who) + ": need at least 3x3x3 nodes");
    if (3 * q.nx * q.ny * q.nz >= (int64_t(1) << 31))
        return fail(SIL_ERR_INVALID, std::string(who) + ": fewer than 2^31 unknowns per problem supported");
    if (q.x == nullptr || q.y == nullptr || q.z == nullptr)
        return fail(SIL_ERR_INVALID, std::string(who) + ": NULL coordinate array");
    if (q.node_mu == nullptr) return fail(SIL_ERR_INVALID, std::string(who) + ": NULL node_mu");
    if (need_fields && (q.rhs == nullptr || q.solution == nullptr))
        return fail(SIL_ERR_INVALID, std::string(who) + ": NULL field pointer");
    if (q.gauge != 0 && q.gauge != 1) return fail(SIL_ERR_INVALID, std::string(who) + ": gauge must be 0 or 1");
    if (!std::isfinite(q.gauge_penalty) || (q.gauge == 0 ? !(q.gauge_penalty > 0.0) : q.gauge_penalty == 0.0))
        return fail(SIL_ERR_INVALID, std::string(who) + ": gauge_penalty must be finite and positive "
                                                        "(nonzero for the divergence gauge)");
    double const* c[3] = {q.x, q.y, q.z};
    int64_t const len[3] = {q.nx, q.ny, q.nz};
    for (int a = 0; a < 3; ++a)
        for (int64_t i = 0; i + 1 < len[a]; ++i)
            if (!(c[a][i + 1] > c[a][i]))
                return fail(SIL_ERR_INVALID, std::string(who) + ": node coordinates must increase strictly");
    return SIL_OK;
}

// A thread per node.  G: the divergence-gauge variant (the penalty variant
// keeps fewer registers).
template <bool G>
__global__ void __launch_bounds__(256, 4) mag3d_apply_kernel(ProbInfo pi, double const* nu, double const* a, double* y)
{
    int64_t const node = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (node >= pi.nodes) return;
    double out[3];
    mag3d_apply_node<double, G>(a, nu, pi, static_cast<int>(node), out);
    for (int c = 0; c < 3; ++c) y[3 * node + c] = out[c];
}

// The penalty operator in marching tiles (mag3d_march.cuh), four CTAs on a
// multiprocessor.
constexpr int kApplyCtas = 4;
__global__ void __launch_bounds__(kMarchThreads, kApplyCtas)
        mag3d_march_kernel(Grid3<double> g, double const* nu, double const* a, double* y, int tiles_x, int tiles_y,
                           int planes)
{
    __shared__ MarchSmem<double> sm;
    int const t = blockIdx.x / tiles_x, bx = blockIdx.x - t * tiles_x, bz = t / tiles_y, by = t - bz * tiles_y;
    int const k0 = bz * planes;
    mag3d_march(sm, g, nu, a, bx * kMarchCols, by * kMarchOwnRows, k0, min(g.nz, k0 + planes),
                [&](int row, double q, double) { y[row] = q; });
}

// Whether the operator marches: from 300,000 nodes on, below which a run's two
// planes of start-up are a tenth or more of the few planes a grid leaves each
// CTA, and where the tiles cover the grid well enough.  A march takes `waves` of
// planes + 2 steps of every resident thread; a thread per node works on the rows
// of interior nodes (a warp of a boundary row ends at once).  Of 58 grids of 0.3
// to 17 M nodes the tiles were the faster ones at three thread steps a node and
// fewer.  B200, thread per node -> tiles, by steps a node: 1.5 256^3 358 -> 218 us
// (4.3 TB/s of the 56 bytes a node; from a CUDA graph), 1.9 250x90x30 17.2 ->
// 12.9, 2.2 96^3 21.7 -> 18.2, 2.8 33x33x1000 30.8 -> 27.9, 3.0 100x60x55 10.6 ->
// 9.9, and beyond: 3.1 40x100x100 13.2 -> 12.9, 3.4 64x64x80 10.9 -> 11.1, 3.8
// 10x1000x1000 300 -> 349, 4.5 2000x8x33 10.8 -> 14.1, 88 3x3x40000 7.1 -> 70.7.
// What bounds the tiles is the data pipe of L1 and shared memory (71 % busy) and
// their issue rate: about 200 instructions per warp and plane at 61 % of the
// issue slots.
constexpr int64_t kMarchMinNodes = 300000;
constexpr int64_t kMarchSteps = 3;   // per interior node

bool mag3d_marches(ProbInfo const& pi, int64_t columns, int planes, int64_t resident)
{
    int64_t const runs = (pi.nz + planes - 1) / planes, waves = (columns * runs + resident - 1) / resident;
    return waves * (planes + 2) * resident * kMarchThreads <= kMarchSteps * pi.nx * (pi.ny - 2) * (pi.nz - 2);
}

sil_status launch_mag3d_apply(ProbInfo const& pi, double const* nu, double const* a, double* y, cudaStream_t s)
{
    unsigned const blocks = static_cast<unsigned>((pi.nodes + 255) / 256);
    int const tx = march_tiles_x(pi), ty = march_tiles_y(pi);
    int64_t const columns = static_cast<int64_t>(tx) * ty, resident = static_cast<int64_t>(kApplyCtas) * multiprocessors();
    int const planes = pi.gauge || pi.nodes < kMarchMinNodes ? 0 : run_length(columns, pi.nz, resident);
    if (pi.gauge) {
        mag3d_apply_kernel<true><<<blocks, 256, 0, s>>>(pi, nu, a, y);
    } else if (planes == 0 || !mag3d_marches(pi, columns, planes, resident)) {
        mag3d_apply_kernel<false><<<blocks, 256, 0, s>>>(pi, nu, a, y);
    } else {
        Grid3<double> const g = march_grid<double>(pi);
        int const runs = (g.nz + planes - 1) / planes;
        mag3d_march_kernel<<<static_cast<unsigned>(tx) * ty * runs, kMarchThreads, 0, s>>>(g, nu, a, y, tx, ty, planes);
    }
    SIL_CUDA_CHECK(cudaGetLastError());
    return SIL_OK;
}

} // namespace

sil_status divergence_gauge_table(int64_t nx, int64_t ny, int64_t nz, double const* const coords[3], double const* ls,
                                  double* gd, double* probe, double* out, cudaStream_t st)
{
    ProblemDesc q {};
    q.dim = 3;
    q.nx = nx;
    q.ny = ny;
    q.nz = nz;
    for (int a = 0; a < 3; ++a) q.coords[a] = coords[a];
    q.gauge = 1;
    ProbInfo pi {};
    pi.dim = 3;
    pi.nx = nx;
    pi.ny = ny;
    pi.nz = nz;
    pi.nodes = nx * ny * nz;
    pi.n = 3 * pi.nodes;
    pi.ls64[0] = ls;
    pi.ls64[1] = ls + nx;
    pi.ls64[2] = ls + nx + ny;
    return build_divergence_gauge(q, pi, gd, nullptr, probe, out, st);
}

} // namespace sil

extern "C" {

sil_status sil_mag3d_apply(sil_stream stream, const sil_mag3d_problem* problem, const double* a, double* y)
{
    if (problem == nullptr || a == nullptr || y == nullptr) return fail(SIL_ERR_INVALID, "sil_mag3d_apply: NULL pointer");
    sil_mag3d_problem const& q = *problem;
    sil_status const st = check_mag3d(q, "sil_mag3d_apply", false);
    if (st != SIL_OK) return st;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    int64_t const nodes = q.nx * q.ny * q.nz;
    int64_t const len[3] = {q.nx, q.ny, q.nz};
    double const* c[3] = {q.x, q.y, q.z};
    std::vector<double> sp;
    for (int a2 = 0; a2 < 3; ++a2)
        for (int64_t i = 0; i < len[a2]; ++i) sp.push_back(local_spacing(c[a2], len[a2], i));
    for (int a2 = 0; a2 < 3; ++a2)
        for (int64_t i = 0; i < len[a2]; ++i) sp.push_back(1.0 / local_spacing(c[a2], len[a2], i));
    size_t const nu_bytes = (nodes * sizeof(double) + 255) / 256 * 256;
    // divergence gauge: coefficient table (8 per node) and probe scratch (3 + 1 per node)
    size_t const gauge_bytes = q.gauge ? static_cast<size_t>(nodes) * 12 * sizeof(double) : 0;
    DeviceBuffer buf;
    SIL_CUDA_CHECK(cudaMallocAsync(&buf.ptr, nu_bytes + gauge_bytes + sp.size() * sizeof(double), s));
    double* nu = static_cast<double*>(buf.ptr);
    double* gd = reinterpret_cast<double*>(static_cast<char*>(buf.ptr) + nu_bytes);
    double* dsp = reinterpret_cast<double*>(static_cast<char*>(buf.ptr) + nu_bytes + gauge_bytes);
    SIL_CUDA_CHECK(cudaMemcpyAsync(dsp, sp.data(), sp.size() * sizeof(double), cudaMemcpyHostToDevice, s));
    ProbInfo pi {};
    pi.dim = 3;
    pi.nx = q.nx;
    pi.ny = q.ny;
    pi.nz = q.nz;
    pi.nodes = nodes;
    pi.n = 3 * nodes;
    pi.gamma = q.gauge_penalty;
    int64_t o = 0;
    for (int a2 = 0; a2 < 3; ++a2) {
        pi.ls64[a2] = dsp + o;
        o += len[a2];
    }
    for (int a2 = 0; a2 < 3; ++a2) {
        pi.ils64[a2] = dsp + o;
        o += len[a2];
    }
    if (q.gauge) {
        ProblemDesc desc {3, q.nx, q.ny, q.nz, q.gauge_penalty, q.node_mu, nullptr, nullptr, {q.x, q.y, q.z}, 1};
        sil_status const gs = build_divergence_gauge(desc, pi, gd, nullptr, gd + 8 * nodes, gd + 11 * nodes, s);
        if (gs != SIL_OK) return gs;
        pi.gauge = 1;
        pi.gd64 = gd;
    }
    reciprocal_kernel<<<static_cast<int>((nodes + 255) / 256), 256, 0, s>>>(q.node_mu, nu, nodes);
    if (sil_status const ls = launch_mag3d_apply(pi, nu, a, y, s); ls != SIL_OK) return ls;
    // A copy from pageable memory has left the host table once it returns;
    // the device buffer is freed in stream order after the apply.
    SIL_CUDA_CHECK(cudaFreeAsync(buf.ptr, s));
    buf.ptr = nullptr;
    return SIL_OK;
}

// A 3D operator with its set-up done once: the device spacing tables, the
// node reluctivity 1/mu and (divergence gauge) the codifferential
// coefficient table, so that an apply is one kernel.
} // extern "C"

struct sil_mag3d_operator_s
{
    sil::ProbInfo pi {};
    double const* nu = nullptr;
    void* mem = nullptr;
};

extern "C" {

sil_status sil_mag3d_operator_create(sil_mag3d_operator* out, sil_stream stream, const sil_mag3d_problem* problem)
{
    if (out == nullptr || problem == nullptr) return fail(SIL_ERR_INVALID, "sil_mag3d_operator_create: NULL pointer");
    *out = nullptr;
    sil_mag3d_problem const& q = *problem;
    sil_status const st = check_mag3d(q, "sil_mag3d_operator_create", false);
    if (st != SIL_OK) return st;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    int64_t const nodes = q.nx * q.ny * q.nz;
    int64_t const len[3] = {q.nx, q.ny, q.nz};
    double const* c[3] = {q.x, q.y, q.z};
    std::vector<double> sp;
    for (int a2 = 0; a2 < 3; ++a2)
        for (int64_t i = 0; i < len[a2]; ++i) sp.push_back(local_spacing(c[a2], len[a2], i));
    for (int a2 = 0; a2 < 3; ++a2)
        for (int64_t i = 0; i < len[a2]; ++i) sp.push_back(1.0 / local_spacing(c[a2], len[a2], i));
    size_t const nu_bytes = (nodes * sizeof(double) + 255) / 256 * 256;
    size_t const gauge_bytes = q.gauge ? static_cast<size_t>(nodes) * 12 * sizeof(double) : 0;
    auto* op = new sil_mag3d_operator_s;
    if (cudaMalloc(&op->mem, nu_bytes + gauge_bytes + sp.size() * sizeof(double)) != cudaSuccess) {
        delete op;
        cudaGetLastError();   // as cuda_fail
        return fail(SIL_ERR_CUDA, "sil_mag3d_operator_create: device allocation failed");
    }
    auto bail = [&](sil_status e) {
        cudaGetLastError();
        cudaFree(op->mem);
        delete op;
        return e;
    };
    double* nu = static_cast<double*>(op->mem);
    double* gd = reinterpret_cast<double*>(static_cast<char*>(op->mem) + nu_bytes);
    double* dsp = reinterpret_cast<double*>(static_cast<char*>(op->mem) + nu_bytes + gauge_bytes);
    if (cudaMemcpyAsync(dsp, sp.data(), sp.size() * sizeof(double), cudaMemcpyHostToDevice, s) != cudaSuccess)
        return bail(fail(SIL_ERR_CUDA, "sil_mag3d_operator_create: table upload failed"));
    ProbInfo& pi = op->pi;
    pi.dim = 3;
    pi.nx = q.nx;
    pi.ny = q.ny;
    pi.nz = q.nz;
    pi.nodes = nodes;
    pi.n = 3 * nodes;
    pi.gamma = q.gauge_penalty;
    int64_t o = 0;
    for (int a2 = 0; a2 < 3; ++a2) {
        pi.ls64[a2] = dsp + o;
        o += len[a2];
    }
    for (int a2 = 0; a2 < 3; ++a2) {
        pi.ils64[a2] = dsp + o;
        o += len[a2];
    }
    if (q.gauge) {
        ProblemDesc desc {3, q.nx, q.ny, q.nz, q.gauge_penalty, q.node_mu, nullptr, nullptr, {q.x, q.y, q.z}, 1};
        sil_status const gs = build_divergence_gauge(desc, pi, gd, nullptr, gd + 8 * nodes, gd + 11 * nodes, s);
        if (gs != SIL_OK) return bail(gs);
        pi.gauge = 1;
        pi.gd64 = gd;
    }
    reciprocal_kernel<<<static_cast<int>((nodes + 255) / 256), 256, 0, s>>>(q.node_mu, nu, nodes);
    if (cudaGetLastError() != cudaSuccess || cudaStreamSynchronize(s) != cudaSuccess)
        return bail(fail(SIL_ERR_CUDA, "sil_mag3d_operator_create: set-up kernels failed"));
    op->nu = nu;
    *out = op;
    return SIL_OK;
}

sil_status sil_mag3d_operator_apply(sil_mag3d_operator op, sil_stream stream, const double* a, double* y)
{
    if (op == nullptr || a == nullptr || y == nullptr) return fail(SIL_ERR_INVALID, "sil_mag3d_operator_apply: NULL pointer");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    return launch_mag3d_apply(op->pi, op->nu, a, y, s);
}

sil_status sil_mag3d_operator_destroy(sil_mag3d_operator op)
{
    if (op == nullptr) return SIL_OK;
    cudaFree(op->mem);
    delete op;
    return SIL_OK;
}

sil_status sil_mag3d_solve_batch(const sil_mag3d_problem* problems, int nproblems, const sil_solve_settings* settings,
                                 sil_solve_diagnostics* diag, sil_stream stream)
{
    if (problems == nullptr || settings == nullptr || diag == nullptr || nproblems < 1)
        return fail(SIL_ERR_INVALID, "sil_mag3d_solve_batch: NULL argument or empty batch");
    std::vector<ProblemDesc> descs(nproblems);
    for (int p = 0; p < nproblems; ++p) {
        sil_mag3d_problem const& q = problems[p];
        sil_status const st = check_mag3d(q, "sil_mag3d_solve_batch", true);
        if (st != SIL_OK) return st;
        descs[p] = {3, q.nx, q.ny, q.nz, q.gauge_penalty, q.node_mu, q.rhs, q.solution, {q.x, q.y, q.z}, q.gauge};
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    std::memset(diag, 0, sizeof(sil_solve_diagnostics) * nproblems);
    sil_chip_limits none = {0, 0, 0, 0};   // nothing of a 3D solve runs on chip
    if (settings->solver == SIL_SOLVER_CG_F64) return solve_batch<double>(descs, *settings, diag, s, none);
    if (settings->solver == SIL_SOLVER_MIXED_IR) return solve_batch<float>(descs, *settings, diag, s, none);
    return fail(SIL_ERR_INVALID, "sil_mag3d_solve_batch: unknown solver kind (the learned solver is 2D only)");
}

} // extern "C"
