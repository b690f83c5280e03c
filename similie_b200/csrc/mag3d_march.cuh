// mag3d_march.cuh -- the 3D curl-curl + penalty-gauge operator over a tile of
// grid columns, marching along z.
//
// A CTA of 32 x 8 threads owns the 31 x 7 columns right of and below its first
// thread column and row, for a run of planes.  Plane by plane it holds the
// operand of planes k and k + 1 in shared memory (a three-slot ring, zero at
// Dirichlet nodes, the slot of plane k + 2 filled by asynchronous copies
// meanwhile), and every thread forms the three weighted curl moments
//   H_m(s) = W_m(s) B_m(s)
// of its node once.  A row of the operator is then four of these moments: the
// node's own, the previous plane's (kept in registers), the left neighbour's
// (a shuffle) and the lower neighbour's (shared memory), so a node costs three
// moments where the node-per-thread kernel forms nine, and its operand loads
// are coalesced (a lane's three components lie 24 bytes apart: read straight
// from global memory each load touches six 128-byte lines).  The moments and
// sums are those of mag3d_curl_rows in the same order, so the values are the
// same.
#pragma once

#include <cstdint>

namespace sil {

// Rectilinear grid of one problem: local spacings and their inverses.
template <class T>
struct Grid3
{
    int nx, ny, nz;
    T gamma;
    T const* l[3];
    T const* il[3];
};

constexpr int kMarchX = 32;            // threads (and columns with a moment) along x
constexpr int kMarchCols = 31;         // owned columns along x
constexpr int kMarchNodes = kMarchX + 1;  // operand nodes along x

// Copies `size` (0: zero-fill) of the sizeof(T) bytes at src to shared memory.
template <class T>
__device__ __forceinline__ void march_copy(T* dst, T const* src, int size)
{
    uint32_t const d = static_cast<uint32_t>(__cvta_generic_to_shared(dst));
    if constexpr (sizeof(T) == 8)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(size) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(size) : "memory");
}
__device__ __forceinline__ void march_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int PENDING>
__device__ __forceinline__ void march_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(PENDING) : "memory");
}

constexpr int kMarchRing = 3;    // operand slots: planes k, k + 1 and the one being filled
constexpr int kMarchWarps = 8;
constexpr int kMarchThreads = kMarchX * kMarchWarps;
constexpr int kMarchOwnRows = kMarchWarps - 1;   // owned columns along y

template <class T>
struct MarchSmem
{
    static constexpr int kElems = (kMarchWarps + 1) * kMarchNodes * 3;
    T a[kMarchRing * kElems];             // operand planes, [slot][row][node][component]
    T h[2 * 2 * kMarchThreads];           // H_x and H_z of the current plane, double-buffered
};

// One run of planes [k0, k1) of the tile whose first owned column is (i0, j0):
// out(row, q, a) takes a result and its operand.  Rows are below 2^31.  EDGE:
// the tile touches the grid's boundary columns, so columns and elements are
// tested; the others test planes only.
template <bool EDGE, class T, class Out>
__device__ __forceinline__ void mag3d_march_tile(MarchSmem<T>& sm, Grid3<T> const& g, T const* __restrict__ nu,
                                                 T const* __restrict__ a, int i0, int j0, int k0, int k1, Out const& out)
{
    constexpr int kRow = kMarchNodes * 3;
    constexpr int kElems = MarchSmem<T>::kElems;
    constexpr int kFull = kElems / kMarchThreads;     // slots every thread fills
    constexpr int kSlots = kFull + (kElems % kMarchThreads != 0);
    int const tid = threadIdx.x, tx = tid & 31, ty = tid >> 5;
    int const i = i0 - 1 + tx, j = j0 - 1 + ty;
    int const nodes2 = g.nx * g.ny, plane = 3 * nodes2;
    bool const tail = tid < kElems % kMarchThreads;   // fills the last, partial slot

    // the elements this thread stages: row offset in a plane, and whether it is
    // an interior one (the others are zero)
    int off[kSlots];
    unsigned inner = 0;
#pragma unroll
    for (int s = 0; s < kSlots; ++s) {
        int const e = min(tid + s * kMarchThreads, kElems - 1), r = e / kRow, c = e - r * kRow;
        int const ii = i0 - 1 + c / 3, jj = j0 - 1 + r;
        bool const deep = !EDGE || (ii > 0 && jj > 0 && ii + 1 < g.nx && jj + 1 < g.ny);
        off[s] = deep ? 3 * (ii + g.nx * jj) + c % 3 : 0;
        if (deep) inner |= 1u << s;
    }
    // Copies of plane k into the ring slot whose first element is `to`.
    auto fetch = [&](int k, int to) {
        if (k <= k1) {
            bool const deep = k > 0 && k + 1 < g.nz;
            T const* from = a + static_cast<int64_t>(plane) * (deep ? k : 0);
#pragma unroll
            for (int s = 0; s < kSlots; ++s)
                if (s < kFull || tail)
                    march_copy(&sm.a[to + tid + s * kMarchThreads], from + off[s],
                               deep && (!EDGE || ((inner >> s) & 1u)) ? static_cast<int>(sizeof(T)) : 0);
        }
        march_commit();
    };

    // the thread's column
    bool const col_in = !EDGE || (i > 0 && j > 0 && i + 1 < g.nx && j + 1 < g.ny);
    bool const col_own = tx > 0 && ty > 0 && (!EDGE || (i < g.nx && j < g.ny));
    int const ic = EDGE ? min(max(i, 0), g.nx - 1) : i, jc = EDGE ? min(max(j, 0), g.ny - 1) : j;
    T const lx = g.l[0][ic], ilx = g.il[0][ic], ly = g.l[1][jc], ily = g.il[1][jc];
    int const node2 = ic + g.nx * jc;

    int slot0 = 0, slot1 = kElems, slot2 = 2 * kElems;   // of planes k, k + 1, k + 2
    fetch(k0 - 1, slot0);
    fetch(k0, slot1);
    fetch(k0 + 1, slot2);
    march_wait<1>();
    __syncthreads();

    int const at = (ty * kMarchNodes + tx) * 3;
    T ax = sm.a[at], ay = sm.a[at + 1], az = sm.a[at + 2], hx_prev = T(0), hy_prev = T(0);
    // the plane's reluctivity and spacing are read a plane early
    T nu_k = nu[node2 + nodes2 * max(k0 - 1, 0)];
    T lz = g.l[2][max(k0 - 1, 0)], ilz = g.il[2][max(k0 - 1, 0)];
    int hs = tid;   // this thread's H_x of the plane
    for (int k = k0 - 1; k < k1; ++k) {
        bool const deep = k > 0 && k + 1 < g.nz;
        int const kn = min(k + 1, k1 - 1);
        T const nu_next = nu[node2 + nodes2 * kn], lz_next = g.l[2][kn], ilz_next = g.il[2][kn];
        T const* A0 = &sm.a[slot0];
        T const* A1 = &sm.a[slot1];
        T const a1x = A1[at], a1y = A1[at + 1], a1z = A1[at + 2];
        // curl moments of node (i, j, k), weighted
        T hx = T(0), hy = T(0), hz = T(0);
        if (deep && col_in) {
            T const Bx = ((ay - az) - a1y) + A0[at + kRow + 2];
            T const By = ((az - ax) + a1x) - A0[at + 3 + 2];
            T const Bz = ((ax - ay) - A0[at + kRow]) + A0[at + 3 + 1];
            hx = (((lx * ily) * ilz) * nu_k) * Bx;
            hy = (((ly * ilx) * ilz) * nu_k) * By;
            hz = (((lz * ilx) * ily) * nu_k) * Bz;
        }
        sm.h[hs] = hx;
        sm.h[hs + kMarchThreads] = hz;
        march_wait<0>();
        __syncthreads();
        // plane k's slot is free now
        fetch(k + kMarchRing, slot0);
        T const hy_left = __shfl_up_sync(0xffffffffu, hy, 1), hz_left = __shfl_up_sync(0xffffffffu, hz, 1);
        T hx_low = T(0), hz_low = T(0);
        if (ty > 0) {
            hx_low = sm.h[hs - kMarchX];
            hz_low = sm.h[hs + kMarchThreads - kMarchX];
        }
        if (k >= k0 && col_own) {
            int const row = 3 * (node2 + nodes2 * k);
            T q0, q1, q2, p0 = ax, p1 = ay, p2 = az;
            if (deep && col_in) {
                q0 = (((hy_prev - hy) + hz) - hz_low) + (g.gamma * ((ly * lz) * ilx)) * ax;
                q1 = (((hx - hx_prev) - hz) + hz_left) + (g.gamma * ((lx * lz) * ily)) * ay;
                q2 = (((hx_low - hx) + hy) - hy_left) + (g.gamma * ((lx * ly) * ilz)) * az;
            } else {
                // identity row of a boundary node: the operand itself
                q0 = p0 = a[row];
                q1 = p1 = a[row + 1];
                q2 = p2 = a[row + 2];
            }
            out(row, q0, p0);
            out(row + 1, q1, p1);
            out(row + 2, q2, p2);
        }
        hs ^= 2 * kMarchThreads;
        hx_prev = hx;
        hy_prev = hy;
        ax = a1x;
        ay = a1y;
        az = a1z;
        nu_k = nu_next;
        lz = lz_next;
        ilz = ilz_next;
        int const t = slot0;
        slot0 = slot1;
        slot1 = slot2;
        slot2 = t;
    }
    march_wait<0>();   // nothing still targets shared memory when the block reuses it or exits
}

template <class T, class Out>
__device__ __forceinline__ void mag3d_march(MarchSmem<T>& sm, Grid3<T> const& g, T const* nu, T const* a, int i0, int j0,
                                            int k0, int k1, Out const& out)
{
    bool const inside = i0 > 1 && j0 > 1 && i0 + kMarchCols < g.nx - 1 && j0 + kMarchOwnRows < g.ny - 1;
    if (inside) mag3d_march_tile<false>(sm, g, nu, a, i0, j0, k0, k1, out);
    else mag3d_march_tile<true>(sm, g, nu, a, i0, j0, k0, k1, out);
}

} // namespace sil
