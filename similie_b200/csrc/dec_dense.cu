// dec_dense.cu -- DEC operators on fields whose lattice is exactly the form
// dims (no spectator dims), 1-3 of them, any strides: d, d^T, the
// codifferential and the fused Hodge Laplacian of every rank, FP64 and FP32.
//
// The table-driven kernels of dec_generic.cu read their sampling rules from
// kernel parameters and keep 64-bit coordinates, so a 3D 1-form Laplacian
// there executes 84 loads per node, each behind a rule fetch, a clamp and a
// multiply per dim.  Here the rank is a template parameter: the rules are
// compile-time constants, the loops unroll completely, equal samples and
// Hodge factors are formed once, and nodes away from the box's edge skip the
// clamps.  Every expression and its order are the table-driven kernel's, so
// the results are the same bits.  What bounds them is the L1 wavefronts of
// loads whose lanes are one node (2-3 components) apart.
//
// Measured on a B200, table-driven -> here: 1-form Laplacian 161x144x130 FP64
// 2,366 -> 145 us, 1999x2741 FP32 1,016 -> 46 us; d + star + codifferential of
// a 150x171x128 1-form FP64 651 -> 122 us (the star is one kernel on both
// sides; the codifferential's march takes it to 112).
#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include <type_traits>

#include "run_plan.cuh"
#include "sil_internal.cuh"

namespace sil {

namespace {

// ------------------------------------------------------------------ rules at compile time

struct Face
{
    int dim;      // the sample is taken at node + shift * e_dim
    int shift;    // -1, 0, +1
    int comp;
    bool negative;
};

constexpr int n_choose(int n, int k)
{
    int r = 1;
    for (int i = 1; i <= k; ++i) r = r * (n - k + i) / i;
    return k < 0 || k > n ? 0 : r;
}

// Index lists of {0..n-1} of size k in lexicographic order, as bit masks.
struct Masks
{
    int count = 0;
    unsigned m[4] = {0, 0, 0, 0};
};

constexpr bool list_less(unsigned a, unsigned b)
{
    for (int d = 0; d < 3; ++d) {
        bool const ia = (a >> d) & 1u, ib = (b >> d) & 1u;
        if (ia != ib) return ia;
    }
    return false;
}

constexpr int bits(unsigned m) { return (m & 1u) + ((m >> 1) & 1u) + ((m >> 2) & 1u); }

constexpr Masks masks(int n, int k)
{
    Masks r {};
    for (unsigned m = 0; m < (1u << n); ++m) {
        if (bits(m) != k) continue;
        int at = r.count;
        while (at > 0 && list_less(m, r.m[at - 1])) {
            r.m[at] = r.m[at - 1];
            --at;
        }
        r.m[at] = m;
        ++r.count;
    }
    return r;
}

constexpr int index_of(Masks const& ms, unsigned m)
{
    for (int i = 0; i < ms.count; ++i)
        if (ms.m[i] == m) return i;
    return -1;
}

// Face f of output component c of d (or d^T) on a k-form over n dims: the
// rule make_rules puts into its table.
constexpr Face face(int n, int k, bool transposed, int c, int f)
{
    int const K = k + 1;
    unsigned const upper = masks(n, K).m[c];
    int const half = f / K, i = f % K;
    int dir = 0;
    for (int d = 0, seen = 0; d < n; ++d) {
        if (!((upper >> d) & 1u)) continue;
        if (seen == i) dir = d;
        ++seen;
    }
    bool const even = K % 2 == 0;
    Face r {};
    r.dim = dir;
    r.comp = index_of(masks(n, k), upper & ~(1u << dir));
    r.shift = half == 0 ? 0 : (transposed ? -1 : 1);
    r.negative = half == 0 ? (((K + i) % 2 == 1) != even) : (((K - 1 + i) % 2 == 1) != even);
    return r;
}

// Diagonal Hodge star of an r-form over n dims, output component t.
struct Star
{
    int src;
    int sgn;
    unsigned num, den;
};

constexpr Star star(int n, int r, int t)
{
    unsigned const out = masks(n, n - r).m[t], c = ((1u << n) - 1) & ~out;
    int inv = 0;
    for (int a = 0; a < n; ++a)
        for (int b = 0; b < a; ++b)
            if (((c >> a) & 1u) && ((out >> b) & 1u)) ++inv;
    return {index_of(masks(n, r), c), inv % 2 ? -1 : 1, out, c};
}

template <int V>
using Int = std::integral_constant<int, V>;

// f(Int<0>{}), ..., f(Int<COUNT - 1>{})
template <int COUNT, int AT = 0, class F>
__device__ __forceinline__ void unroll(F const& f)
{
    if constexpr (AT < COUNT) {
        f(Int<AT> {});
        unroll<COUNT, AT + 1>(f);
    }
}

// ------------------------------------------------------------------ fields

// Coordinates are local to the input box.
template <class T, int N>
struct Dense
{
    T const* in;
    T* out;
    T const* h[N];    // edge lengths by input coordinate
    T const* ih[N];   // and their inverses
    int iext[N], istr[N], ics;
    int oext[N], ostr[N], ocs;
    int off[N];       // output front - input front
    uint32_t total;
};

template <int N>
struct Coord
{
    int v[N];
};

template <int DIM, int SHIFT, int N>
__device__ __forceinline__ Coord<N> moved(Coord<N> c)
{
    c.v[DIM] += SHIFT;
    return c;
}

template <class T, int N>
__device__ __forceinline__ T load(Dense<T, N> const& a, Coord<N> const& c, int comp)
{
    int o = comp * a.ics;
#pragma unroll
    for (int d = 0; d < N; ++d) o += c.v[d] * a.istr[d];
    return __ldg(a.in + o);
}

// DEEP: every sample the operator takes lies in the box.
template <bool DEEP, class T, int N>
__device__ __forceinline__ bool in_box(Dense<T, N> const& a, Coord<N> const& c)
{
    if constexpr (DEEP) return true;
    bool in = true;
#pragma unroll
    for (int d = 0; d < N; ++d) in = in && c.v[d] >= 0 && c.v[d] < a.iext[d];
    return in;
}

template <bool DEEP, class T, int N>
__device__ __forceinline__ Coord<N> clamped(Dense<T, N> const& a, Coord<N> c)
{
    if constexpr (!DEEP) {
#pragma unroll
        for (int d = 0; d < N; ++d) c.v[d] = min(max(c.v[d], 0), a.iext[d] - 1);
    }
    return c;
}

// sign * product of edge lengths over num * product of inverse lengths over den.
template <int R, int TT, class T, int N>
__device__ __forceinline__ T star_factor(Dense<T, N> const& a, Coord<N> const& c)
{
    T f = static_cast<T>(star(N, R, TT).sgn);
    unroll<N>([&](auto d) {
        constexpr int D = decltype(d)::value;
        constexpr Star s = star(N, R, TT);
        if constexpr ((s.num >> D) & 1u) f *= __ldg(a.h[D] + c.v[D]);
        if constexpr ((s.den >> D) & 1u) f *= __ldg(a.ih[D] + c.v[D]);
    });
    return f;
}

// ------------------------------------------------------------------ operators at a node

// Chain-order signed sum over the faces of output component C of d / d^T on
// an R-form; v(coord, comp) samples the form.
template <int N, int R, bool TR, int C, class T, class V>
__device__ __forceinline__ T chain(Coord<N> const& c, V const& v)
{
    T acc = T(0);
    unroll<2 * (R + 1)>([&](auto f) {
        constexpr Face r = face(N, R, TR, C, decltype(f)::value);
        T const s = v(moved<r.dim, r.shift>(c), Int<r.comp> {});
        acc = r.negative ? acc - s : acc + s;
    });
    return acc;
}

// Component C of d of the K-form input (clamped samples).
template <int K, int C, bool DEEP, class T, int N>
__device__ __forceinline__ T d_at(Dense<T, N> const& a, Coord<N> const& c)
{
    return chain<N, K, false, C, T>(c, [&](Coord<N> s, auto comp) {
        return load(a, clamped<DEEP>(a, s), decltype(comp)::value);
    });
}

// Component C of d^T of the K-form input (zero outside).
template <int K, int C, bool DEEP, class T, int N>
__device__ __forceinline__ T dt_at(Dense<T, N> const& a, Coord<N> const& c)
{
    return -chain<N, K, true, C, T>(c, [&](Coord<N> s, auto comp) {
        return in_box<DEEP>(a, s) ? load(a, s, decltype(comp)::value) : T(0);
    });
}

template <int N, int K, class T>
constexpr T delta_sign()
{
    return ((N * (K + 1) + 1) % 2) ? T(-1) : T(1);
}

// Component TT of the codifferential of the K-form input.
template <int K, int TT, bool DEEP, class T, int N>
__device__ __forceinline__ T codiff_at(Dense<T, N> const& a, Coord<N> const& p)
{
    constexpr Star st = star(N, N - K + 1, TT);
    T const acc = chain<N, N - K, true, st.src, T>(p, [&](Coord<N> s, auto comp) {
        constexpr int C = decltype(comp)::value;
        return in_box<DEEP>(a, s) ? star_factor<K, C>(a, s) * load(a, s, star(N, K, C).src) : T(0);
    });
    T const dual = -acc;
    return delta_sign<N, K, T>() * (star_factor<N - K + 1, TT>(a, p) * dual);
}

// Component TT of (delta d + d delta) of the K-form input.
template <int K, int TT, bool DEEP, class T, int N>
__device__ __forceinline__ T laplacian_at(Dense<T, N> const& a, Coord<N> const& p)
{
    T result = T(0);
    if constexpr (K < N) {
        constexpr Star st = star(N, N - K, TT);
        T const acc = chain<N, N - K - 1, true, st.src, T>(p, [&](Coord<N> s, auto comp) {
            // the star of d at s, zero outside the input
            constexpr int C = decltype(comp)::value;
            if (!in_box<DEEP>(a, s)) return T(0);
            T const dv = d_at<K, star(N, K + 1, C).src, DEEP>(a, s);
            return star_factor<K + 1, C>(a, s) * dv;
        });
        T const dual = -acc;
        result = delta_sign<N, K + 1, T>() * (star_factor<N - K, TT>(a, p) * dual);
    }
    if constexpr (K > 0) {
        T const acc = chain<N, K - 1, false, TT, T>(p, [&](Coord<N> s, auto comp) {
            return codiff_at<K, decltype(comp)::value, DEEP>(a, clamped<DEEP>(a, s));
        });
        result = K < N ? result + acc : acc;
    }
    return result;
}

enum Op { kD = 0, kDT = 1, kCodiff = 2, kLaplacian = 3 };

template <int OP, int N, int K>
constexpr int out_comps()
{
    return n_choose(N, OP == kLaplacian ? K : (OP == kCodiff ? K - 1 : K + 1));
}

template <int OP, int K, bool DEEP, class T, int N>
__device__ __forceinline__ void node(Dense<T, N> const& a, Coord<N> const& c, T* o)
{
    unroll<out_comps<OP, N, K>()>([&](auto t) {
        constexpr int TT = decltype(t)::value;
        T v;
        if constexpr (OP == kD) v = d_at<K, TT, DEEP>(a, c);
        else if constexpr (OP == kDT) v = dt_at<K, TT, DEEP>(a, c);
        else if constexpr (OP == kCodiff) v = codiff_at<K, TT, DEEP>(a, c);
        else v = laplacian_at<K, TT, DEEP>(a, c);
        o[TT * a.ocs] = v;
    });
}

constexpr int kDenseBlock = 128;

// One thread per output node, the last dim fastest.
template <int OP, int K, class T, int N>
__global__ void __launch_bounds__(kDenseBlock) dense_kernel(const __grid_constant__ Dense<T, N> a)
{
    uint32_t const flat = blockIdx.x * static_cast<uint32_t>(kDenseBlock) + threadIdx.x;
    if (flat >= a.total) return;
    Coord<N> c;
    T* o = a.out;
    {
        uint32_t r = flat;
        int off = 0;
#pragma unroll
        for (int d = N - 1; d >= 0; --d) {
            int l = static_cast<int>(r);
            if (d > 0) {
                uint32_t const e = static_cast<uint32_t>(a.oext[d]), q = r / e;
                l = static_cast<int>(r - q * e);
                r = q;
            }
            c.v[d] = l + a.off[d];
            off += l * a.ostr[d];
        }
        o += off;
    }
    bool deep = true;
#pragma unroll
    for (int d = 0; d < N; ++d) deep = deep && c.v[d] > 0 && c.v[d] + 1 < a.iext[d];
    if (deep) node<OP, K, true>(a, c, o);
    else node<OP, K, false>(a, c, o);
}

// ------------------------------------------------------------------ marching Laplacians
//
// The Laplacian as its chain of point-wise stages, marched along the slowest
// dim (x) so that each stage's value is formed once per node and handed to the
// neighbours that need it:
//   S = star_k w              at every node, zero outside the box
//   D = star_{k+1} d w        at every node, zero outside (d samples clamped)
//   E = codifferential        from S at the node and one node back per dim
//   result = sign (star d^T D) + d E, D one node back, E one node on (clamped)
// A thread owns one (y, z) column (a lane of one y column in 2D); the x
// neighbours are its own values of the previous and next plane.  Each stage is
// the per-node kernel's expression in the same order: the same bits.  Output
// boxes that reach outside the input keep the per-node kernel.
//
// B200, per-node kernel -> march: 3D 1-form 161x144x130 FP64 143 -> 54 us (2.7
// TB/s), FP32 107 -> 38; 2D 1-form 1999x2741 FP32 46 -> 21 us (4.1 TB/s, its
// fields in L2; 28 when they are not).  The 3D march is bound by the data pipe
// of L1 and shared memory (68 % busy), its instructions (58 % of the issue slots)
// and the 30 % of its threads that only serve their neighbours, the 2D one by
// the loads its sixteen warps a multiprocessor have in flight.

// Chain-order sum like chain(), the sampler taking the face's dim and shift.
template <int N, int R, bool TR, int C, class T, class V>
__device__ __forceinline__ T chain_of(V const& v)
{
    T acc = T(0);
    unroll<2 * (R + 1)>([&](auto f) {
        constexpr Face r = face(N, R, TR, C, decltype(f)::value);
        T const s = v(Int<r.dim> {}, Int<r.shift> {}, Int<r.comp> {});
        acc = r.negative ? acc - s : acc + s;
    });
    return acc;
}

template <int R, int TT, class T, int N>
__device__ __forceinline__ T star_product(T const (&h)[N], T const (&ih)[N])
{
    T f = static_cast<T>(star(N, R, TT).sgn);
    unroll<N>([&](auto d) {
        constexpr int D = decltype(d)::value;
        constexpr Star s = star(N, R, TT);
        if constexpr ((s.num >> D) & 1u) f *= h[D];
        if constexpr ((s.den >> D) & 1u) f *= ih[D];
    });
    return f;
}

template <int N, int K>
struct Stages
{
    static constexpr int kIn = n_choose(N, K);                          // w, S and the result
    static constexpr int kD = K < N ? n_choose(N, N - K - 1) : 0;       // D
    static constexpr int kE = K > 0 ? n_choose(N, K - 1) : 0;           // E
};

// A 1 x N array of values per stage, never empty.
template <class T, int COUNT>
struct Vals
{
    T v[COUNT > 0 ? COUNT : 1];
};

template <int N, int K, class T>
__device__ __forceinline__ Vals<T, Stages<N, K>::kIn> stage_s(Vals<T, Stages<N, K>::kIn> const& w, T const (&h)[N],
                                                              T const (&ih)[N], bool inside)
{
    Vals<T, Stages<N, K>::kIn> s;
    unroll<n_choose(N, N - K)>([&](auto c) {
        constexpr int C = decltype(c)::value;
        s.v[C] = inside ? star_product<K, C>(h, ih) * w.v[star(N, K, C).src] : T(0);
    });
    return s;
}

// W(dim, shift, comp): w at the node + shift e_dim.
template <int N, int K, class T, class W>
__device__ __forceinline__ Vals<T, Stages<N, K>::kD> stage_d(W const& w, T const (&h)[N], T const (&ih)[N], bool inside)
{
    Vals<T, Stages<N, K>::kD> d;
    if constexpr (K < N)
        unroll<Stages<N, K>::kD>([&](auto c) {
            constexpr int C = decltype(c)::value;
            T const dv = chain_of<N, K, false, star(N, K + 1, C).src, T>(w);
            d.v[C] = inside ? star_product<K + 1, C>(h, ih) * dv : T(0);
        });
    return d;
}

// S(dim, shift, comp): S at the node + shift e_dim.
template <int N, int K, class T, class W>
__device__ __forceinline__ Vals<T, Stages<N, K>::kE> stage_e(W const& sv, T const (&h)[N], T const (&ih)[N])
{
    Vals<T, Stages<N, K>::kE> e;
    if constexpr (K > 0)
        unroll<Stages<N, K>::kE>([&](auto t) {
            constexpr int TT = decltype(t)::value;
            T const dual = -chain_of<N, N - K, true, star(N, N - K + 1, TT).src, T>(sv);
            e.v[TT] = delta_sign<N, K, T>() * (star_product<N - K + 1, TT>(h, ih) * dual);
        });
    return e;
}

// D and E samplers as above; result component TT.
template <int N, int K, int TT, class T, class DV, class EV>
__device__ __forceinline__ T stage_result(DV const& dv, EV const& ev, T const (&h)[N], T const (&ih)[N])
{
    T result = T(0);
    if constexpr (K < N) {
        T const dual = -chain_of<N, N - K - 1, true, star(N, N - K, TT).src, T>(dv);
        result = delta_sign<N, K + 1, T>() * (star_product<N - K, TT>(h, ih) * dual);
    }
    if constexpr (K > 0) {
        T const acc = chain_of<N, K - 1, false, TT, T>(ev);
        result = K < N ? result + acc : acc;
    }
    return result;
}

// ---- 3D: a CTA of 32 x MARCH_Y threads owns the 30 x (MARCH_Y - 2) inner
// columns (z along the lanes).  The form's planes arrive by asynchronous copies
// of whole rows, coalesced whatever the component count, into a three-slot
// ring; S, D and E pass between threads through double-buffered planes with one
// barrier a plane.
constexpr int kMarchZ = 32;

__device__ __forceinline__ void copy_async(void* dst, void const* src, Int<8>)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
                 "l"(src)
                 : "memory");
}
__device__ __forceinline__ void copy_async(void* dst, void const* src, Int<4>)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))),
                 "l"(src)
                 : "memory");
}

template <class T, int K, int Y>
struct Lap3Smem
{
    using St = Stages<3, K>;
    static constexpr int kThreads = kMarchZ * Y;
    T w[3][Y * kMarchZ * St::kIn];
    T s[K > 0 ? 2 : 1][K > 0 ? St::kIn : 1][kThreads];
    T d[K < 3 ? 2 : 1][K < 3 ? St::kD : 1][kThreads];
    T e[K > 0 ? 2 : 1][K > 0 ? St::kE : 1][kThreads];
};

template <class T, int K, int Y, int CTAS>
__global__ void __launch_bounds__(kMarchZ* Y, CTAS)
        lap3_march_kernel(const __grid_constant__ Dense<T, 3> a, int tiles_z, int tiles_y, int planes)
{
    using St = Stages<3, K>;
    constexpr int kThreads = kMarchZ * Y, kRow = kMarchZ * St::kIn, kSlots = St::kIn;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    auto& sm = *reinterpret_cast<Lap3Smem<T, K, Y>*>(smem_raw);
    int const tid = threadIdx.x, tz = tid & 31, ty = tid >> 5;
    int const t = blockIdx.x / tiles_z, bz = blockIdx.x - t * tiles_z, bx = t / tiles_y, by = t - bx * tiles_y;
    // first owned output column, and the input coordinates of this thread's column
    int const oz = bz * (kMarchZ - 2), oy = by * (Y - 2), ox0 = bx * planes, ox1 = min(a.oext[0], ox0 + planes);
    int const z = oz + a.off[2] - 1 + tz, y = oy + a.off[1] - 1 + ty;
    int const X = a.iext[0], Ny = a.iext[1], Nz = a.iext[2];
    auto clampi = [](int v, int n) { return min(max(v, 0), n - 1); };
    bool const col_in = z >= 0 && y >= 0 && z < Nz && y < Ny;
    bool const own = tz > 0 && ty > 0 && tz < kMarchZ - 1 && ty < Y - 1 && oz + tz - 1 < a.oext[2] && oy + ty - 1 < a.oext[1];
    // neighbour threads for E one node on, the last node of the box its own (clamped)
    int const next_z = z + 1 < Nz ? tid + 1 : tid, next_y = y + 1 < Ny ? tid + kMarchZ : tid;
    // The elements this thread copies: kSlots runs of kThreads consecutive
    // tile elements; a node past the box is the clamped one.
    int src[kSlots];
#pragma unroll
    for (int q = 0; q < kSlots; ++q) {
        int const e = tid + q * kThreads, r = e / kRow, c = e - r * kRow;
        src[q] = clampi(oy + a.off[1] - 1 + r, Ny) * a.istr[1]
                 + clampi(oz + a.off[2] - 1 + c / St::kIn, Nz) * a.istr[2] + c % St::kIn * a.ics;
    }
    auto fetch = [&](int x, int slot) {
        T const* plane = a.in + static_cast<int64_t>(clampi(x, X)) * a.istr[0];
#pragma unroll
        for (int q = 0; q < kSlots; ++q)
            copy_async(&sm.w[slot][tid + q * kThreads], plane + src[q], Int<static_cast<int>(sizeof(T))> {});
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    T h[3], ih[3], h_on[3], ih_on[3];
    h[1] = h_on[1] = __ldg(a.h[1] + clampi(y, Ny));
    ih[1] = ih_on[1] = __ldg(a.ih[1] + clampi(y, Ny));
    h[2] = h_on[2] = __ldg(a.h[2] + clampi(z, Nz));
    ih[2] = ih_on[2] = __ldg(a.ih[2] + clampi(z, Nz));

    // march from one plane before the first output (its D and the E after it)
    int const x_first = ox0 + a.off[0] - 1, x_last = ox1 - 1 + a.off[0];
    fetch(x_first, 0);
    fetch(x_first + 1, 1);
    fetch(x_first + 2, 2);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    int const at = tid * St::kIn;
    Vals<T, St::kIn> w0, s0;
    Vals<T, St::kD> d_back;
    Vals<T, St::kE> e0;
    int slot0 = 0, slot1 = 1, slot2 = 2;
    h[0] = __ldg(a.h[0] + clampi(x_first, X));
    ih[0] = __ldg(a.ih[0] + clampi(x_first, X));
#pragma unroll
    for (int c = 0; c < St::kIn; ++c) w0.v[c] = sm.w[0][at + c];
    s0 = stage_s<3, K, T>(w0, h, ih, col_in && x_first >= 0 && x_first < X);
#pragma unroll
    for (int c = 0; c < St::kD; ++c) d_back.v[c] = T(0);
#pragma unroll
    for (int c = 0; c < St::kE; ++c) e0.v[c] = T(0);
    for (int x = x_first; x <= x_last; ++x) {
        int const buf = x & 1;
        bool const in0 = col_in && x >= 0 && x < X, in1 = col_in && x + 1 >= 0 && x + 1 < X;
        h_on[0] = __ldg(a.h[0] + clampi(x + 1, X));
        ih_on[0] = __ldg(a.ih[0] + clampi(x + 1, X));
        Vals<T, St::kIn> w1, s1;
#pragma unroll
        for (int c = 0; c < St::kIn; ++c) w1.v[c] = sm.w[slot1][at + c];
        T const* plane = sm.w[slot0];
        // the last column of a tile row and the last row hold no D that is used
        int const up_z = tz < kMarchZ - 1 ? at + St::kIn : at, up_y = ty < Y - 1 ? at + kRow : at;
        Vals<T, St::kD> const d0 = stage_d<3, K, T>(
                [&](auto dim, auto shift, auto comp) -> T {
                    constexpr int C = decltype(comp)::value;
                    if constexpr (decltype(shift)::value == 0) return w0.v[C];
                    else if constexpr (decltype(dim)::value == 0) return w1.v[C];
                    else if constexpr (decltype(dim)::value == 1) return plane[up_y + C];
                    else return plane[up_z + C];
                },
                h, ih, in0);
        s1 = stage_s<3, K, T>(w1, h_on, ih_on, in1);
        if constexpr (K > 0)
#pragma unroll
            for (int c = 0; c < St::kIn; ++c) sm.s[buf][c][tid] = s1.v[c];
        if constexpr (K < 3)
#pragma unroll
            for (int c = 0; c < St::kD; ++c) sm.d[buf][c][tid] = d0.v[c];
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();
        // every thread is past plane x's slot: plane x + 3 takes it
        if (x + 2 <= x_last) fetch(x + 3, slot0);
        int const back_z = tz > 0 ? tid - 1 : tid, back_y = ty > 0 ? tid - kMarchZ : tid;
        Vals<T, St::kE> const e_new = stage_e<3, K, T>(
                [&](auto dim, auto shift, auto comp) -> T {
                    constexpr int C = decltype(comp)::value;
                    if constexpr (decltype(shift)::value == 0) return s1.v[C];
                    else if constexpr (decltype(dim)::value == 0) return s0.v[C];
                    else if constexpr (decltype(dim)::value == 1) return sm.s[K > 0 ? buf : 0][K > 0 ? C : 0][back_y];
                    else return sm.s[K > 0 ? buf : 0][K > 0 ? C : 0][back_z];
                },
                h_on, ih_on);
        Vals<T, St::kE> const e1 = x + 1 < X ? e_new : e0;   // clamped at the last plane
        if constexpr (K > 0)
#pragma unroll
            for (int c = 0; c < St::kE; ++c) sm.e[buf ^ 1][c][tid] = e1.v[c];
        if (x > x_first && own) {
            T* o = a.out + static_cast<int64_t>(x - a.off[0]) * a.ostr[0] + (oy + ty - 1) * a.ostr[1]
                   + (oz + tz - 1) * a.ostr[2];
            unroll<St::kIn>([&](auto tt) {
                constexpr int TT = decltype(tt)::value;
                T const v = stage_result<3, K, TT, T>(
                        [&](auto dim, auto shift, auto comp) -> T {
                            constexpr int C = decltype(comp)::value;
                            if constexpr (decltype(shift)::value == 0) return d0.v[C];
                            else if constexpr (decltype(dim)::value == 0) return d_back.v[C];
                            else if constexpr (decltype(dim)::value == 1) return sm.d[K < 3 ? buf : 0][K < 3 ? C : 0][back_y];
                            else return sm.d[K < 3 ? buf : 0][K < 3 ? C : 0][back_z];
                        },
                        [&](auto dim, auto shift, auto comp) -> T {
                            constexpr int C = decltype(comp)::value;
                            if constexpr (decltype(shift)::value == 0) return e0.v[C];
                            else if constexpr (decltype(dim)::value == 0) return e1.v[C];
                            else if constexpr (decltype(dim)::value == 1) return sm.e[K > 0 ? buf : 0][K > 0 ? C : 0][next_y];
                            else return sm.e[K > 0 ? buf : 0][K > 0 ? C : 0][next_z];
                        },
                        h, ih);
                o[TT * a.ocs] = v;
            });
        }
        d_back = d0;
        e0 = e1;
        s0 = s1;
        w0 = w1;
        h[0] = h_on[0];
        ih[0] = ih_on[0];
        int const q = slot0;
        slot0 = slot1;
        slot1 = slot2;
        slot2 = q;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// The 3D codifferential, marched the same way: S from the ring's plane, its y
// and z neighbours through a double-buffered plane, its x neighbour kept.  Only
// lower neighbours are read, so the tile owns 31 x (Y - 1) columns.
//
// Bound by the data pipe of L1 and shared memory (65 % busy, half of its shared
// wavefronts bank conflicts of the three-component ring) and the idle threads of
// its tiles; 63 % of the copy rate at 150x171x128, FP64.  B200, node kernel ->
// march at that size: 2-form FP64 52.8 -> 39.8 us, FP32 47.2 -> 27.5; 1-form 34.5
// -> 30.1, 32.0 -> 24.1; 3-form 36.2 -> 30.2, 33.4 -> 20.1.
template <class T, int K, int Y>
struct Codiff3Smem
{
    T w[3][Y * kMarchZ * Stages<3, K>::kIn];
    T s[2][Stages<3, K>::kIn][kMarchZ * Y];
};

template <class T, int K, int Y, int CTAS>
__global__ void __launch_bounds__(kMarchZ* Y, CTAS)
        codiff3_march_kernel(const __grid_constant__ Dense<T, 3> a, int tiles_z, int tiles_y, int planes)
{
    using St = Stages<3, K>;
    constexpr int kThreads = kMarchZ * Y, kRow = kMarchZ * St::kIn, kSlots = St::kIn;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    auto& sm = *reinterpret_cast<Codiff3Smem<T, K, Y>*>(smem_raw);
    int const tid = threadIdx.x, tz = tid & 31, ty = tid >> 5;
    int const t = blockIdx.x / tiles_z, bz = blockIdx.x - t * tiles_z, bx = t / tiles_y, by = t - bx * tiles_y;
    int const oz = bz * (kMarchZ - 1), oy = by * (Y - 1), ox0 = bx * planes, ox1 = min(a.oext[0], ox0 + planes);
    int const z = oz + a.off[2] - 1 + tz, y = oy + a.off[1] - 1 + ty;
    int const X = a.iext[0], Ny = a.iext[1], Nz = a.iext[2];
    auto clampi = [](int v, int n) { return min(max(v, 0), n - 1); };
    bool const col_in = z >= 0 && y >= 0 && z < Nz && y < Ny;
    bool const own = tz > 0 && ty > 0 && oz + tz - 1 < a.oext[2] && oy + ty - 1 < a.oext[1];
    int src[kSlots];
#pragma unroll
    for (int q = 0; q < kSlots; ++q) {
        int const e = tid + q * kThreads, r = e / kRow, c = e - r * kRow;
        src[q] = clampi(oy + a.off[1] - 1 + r, Ny) * a.istr[1]
                 + clampi(oz + a.off[2] - 1 + c / St::kIn, Nz) * a.istr[2] + c % St::kIn * a.ics;
    }
    int const x_first = ox0 + a.off[0] - 1, x_last = ox1 - 1 + a.off[0];
    auto fetch = [&](int x, int slot) {
        if (x <= x_last) {
            T const* plane = a.in + static_cast<int64_t>(clampi(x, X)) * a.istr[0];
#pragma unroll
            for (int q = 0; q < kSlots; ++q)
                copy_async(&sm.w[slot][tid + q * kThreads], plane + src[q], Int<static_cast<int>(sizeof(T))> {});
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch(x_first, 0);
    fetch(x_first + 1, 1);
    fetch(x_first + 2, 2);
    T h[3], ih[3];
    h[1] = __ldg(a.h[1] + clampi(y, Ny));
    ih[1] = __ldg(a.ih[1] + clampi(y, Ny));
    h[2] = __ldg(a.h[2] + clampi(z, Nz));
    ih[2] = __ldg(a.ih[2] + clampi(z, Nz));
    asm volatile("cp.async.wait_group 2;" ::: "memory");
    __syncthreads();
    int const at = tid * St::kIn, back_z = tz > 0 ? tid - 1 : tid, back_y = ty > 0 ? tid - kMarchZ : tid;
    T* o = a.out + static_cast<int64_t>(ox0) * a.ostr[0] + (oy + ty - 1) * a.ostr[1] + (oz + tz - 1) * a.ostr[2];
    Vals<T, St::kIn> s0;
#pragma unroll
    for (int c = 0; c < St::kIn; ++c) s0.v[c] = T(0);
    int slot0 = 0, slot1 = 1, slot2 = 2;
    for (int x = x_first; x <= x_last; ++x) {
        int const buf = x & 1;
        h[0] = __ldg(a.h[0] + clampi(x, X));
        ih[0] = __ldg(a.ih[0] + clampi(x, X));
        Vals<T, St::kIn> w;
#pragma unroll
        for (int c = 0; c < St::kIn; ++c) w.v[c] = sm.w[slot0][at + c];
        Vals<T, St::kIn> const s1 = stage_s<3, K, T>(w, h, ih, col_in && x >= 0 && x < X);
#pragma unroll
        for (int c = 0; c < St::kIn; ++c) sm.s[buf][c][tid] = s1.v[c];
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        // every thread is past plane x's slot: plane x + 3 takes it
        fetch(x + 3, slot0);
        if (x > x_first && own) {
            Vals<T, St::kE> const e = stage_e<3, K, T>(
                    [&](auto dim, auto shift, auto comp) -> T {
                        constexpr int C = decltype(comp)::value;
                        if constexpr (decltype(shift)::value == 0) return s1.v[C];
                        else if constexpr (decltype(dim)::value == 0) return s0.v[C];
                        else if constexpr (decltype(dim)::value == 1) return sm.s[buf][C][back_y];
                        else return sm.s[buf][C][back_z];
                    },
                    h, ih);
#pragma unroll
            for (int c = 0; c < St::kE; ++c) o[c * a.ocs] = e.v[c];
            o += a.ostr[0];
        }
        s0 = s1;
        int const q = slot0;
        slot0 = slot1;
        slot1 = slot2;
        slot2 = q;
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
}

// ---- 2D 1-forms: a warp per strip of 30 owned columns (y along the lanes), no
// shared memory: the y neighbours' values come from the next lanes.  Four
// planes' loads are in flight before the first is used.
constexpr int kStripOwn = 30, kStripBatch = 4, kStripThreads = 256;

template <class T, bool VEC>
__global__ void __launch_bounds__(kStripThreads, 2)
        lap2_strip_kernel(const __grid_constant__ Dense<T, 2> a, int strips, int rows)
{
    constexpr int K = 1, U = kStripBatch;
    using St = Stages<2, K>;
    using T2 = std::conditional_t<sizeof(T) == 8, double2, float2>;
    int const lane = threadIdx.x & 31;
    int const cta_strips = kStripThreads / 32, groups = (strips + cta_strips - 1) / cta_strips;
    int const bx = blockIdx.x / groups, strip = (blockIdx.x - bx * groups) * cta_strips + static_cast<int>(threadIdx.x >> 5);
    if (strip >= strips) return;
    int const X = a.iext[0], Ny = a.iext[1];
    int const oy = strip * kStripOwn, y = oy + a.off[1] - 1 + lane;
    int const ox0 = bx * rows, ox1 = min(a.oext[0], ox0 + rows);
    auto clampi = [](int v, int n) { return min(max(v, 0), n - 1); };
    int const yc = clampi(y, Ny);
    bool const col_in = y >= 0 && y < Ny;
    bool const own = lane > 0 && lane <= kStripOwn && oy + lane - 1 < a.oext[1];
    T const* col = a.in + yc * a.istr[1];
    auto load_w = [&](int x) {
        T const* p = col + static_cast<int64_t>(clampi(x, X)) * a.istr[0];
        Vals<T, 2> w;
        if constexpr (VEC) {
            T2 const v = __ldg(reinterpret_cast<T2 const*>(p));
            w.v[0] = v.x;
            w.v[1] = v.y;
        } else {
            w.v[0] = __ldg(p);
            w.v[1] = __ldg(p + a.ics);
        }
        return w;
    };
    T h[2], ih[2], h_on[2], ih_on[2];
    h[1] = h_on[1] = __ldg(a.h[1] + yc);
    ih[1] = ih_on[1] = __ldg(a.ih[1] + yc);
    int const x_first = ox0 + a.off[0] - 1, x_last = ox1 - 1 + a.off[0];
    Vals<T, 2> w0 = load_w(x_first), s0;
    h[0] = __ldg(a.h[0] + clampi(x_first, X));
    ih[0] = __ldg(a.ih[0] + clampi(x_first, X));
    T d_back = T(0), e0 = T(0);
    T* out = a.out + static_cast<int64_t>(ox0 - 1) * a.ostr[0] + (oy + lane - 1) * a.ostr[1];
    for (int xb = x_first; xb <= x_last; xb += U) {
        Vals<T, 2> w[U];
        T hx[U], ihx[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            w[u] = load_w(xb + 1 + u);
            hx[u] = __ldg(a.h[0] + clampi(xb + 1 + u, X));
            ihx[u] = __ldg(a.ih[0] + clampi(xb + 1 + u, X));
        }
        if (xb == x_first) s0 = stage_s<2, K, T>(w0, h, ih, col_in && x_first >= 0 && x_first < X);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            int const x = xb + u;
            bool const in0 = col_in && x >= 0 && x < X, in1 = col_in && x + 1 >= 0 && x + 1 < X;
            h_on[0] = hx[u];
            ih_on[0] = ihx[u];
            Vals<T, 2> const w1 = w[u];
            Vals<T, 2> const s1 = stage_s<2, K, T>(w1, h_on, ih_on, in1);
            Vals<T, 2> up, back;
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                up.v[c] = __shfl_down_sync(0xffffffffu, w0.v[c], 1);
                back.v[c] = __shfl_up_sync(0xffffffffu, s1.v[c], 1);
            }
            T const d0 = stage_d<2, K, T>(
                                 [&](auto dim, auto shift, auto comp) -> T {
                                     constexpr int C = decltype(comp)::value;
                                     if constexpr (decltype(shift)::value == 0) return w0.v[C];
                                     else if constexpr (decltype(dim)::value == 0) return w1.v[C];
                                     else return up.v[C];
                                 },
                                 h, ih, in0)
                                 .v[0];
            T const e_new = stage_e<2, K, T>(
                                    [&](auto dim, auto shift, auto comp) -> T {
                                        constexpr int C = decltype(comp)::value;
                                        if constexpr (decltype(shift)::value == 0) return s1.v[C];
                                        else if constexpr (decltype(dim)::value == 0) return s0.v[C];
                                        else return back.v[C];
                                    },
                                    h_on, ih_on)
                                    .v[0];
            T const e1 = x + 1 < X ? e_new : e0;   // clamped at the last plane
            T const d_left = __shfl_up_sync(0xffffffffu, d0, 1);
            T const e_next = __shfl_down_sync(0xffffffffu, e0, 1), e_right = y + 1 < Ny ? e_next : e0;
            T r[2];
            unroll<2>([&](auto tt) {
                constexpr int TT = decltype(tt)::value;
                r[TT] = stage_result<2, K, TT, T>(
                        [&](auto dim, auto shift, auto) -> T {
                            if constexpr (decltype(shift)::value == 0) return d0;
                            else if constexpr (decltype(dim)::value == 0) return d_back;
                            else return d_left;
                        },
                        [&](auto dim, auto shift, auto) -> T {
                            if constexpr (decltype(shift)::value == 0) return e0;
                            else if constexpr (decltype(dim)::value == 0) return e1;
                            else return e_right;
                        },
                        h, ih);
            });
            if (own && x > x_first && x <= x_last) {
                T* o = out + static_cast<int64_t>(x - x_first) * a.ostr[0];
                if constexpr (VEC) {
                    T2 v;
                    v.x = r[0];
                    v.y = r[1];
                    *reinterpret_cast<T2*>(o) = v;
                } else {
                    o[0] = r[0];
                    o[a.ocs] = r[1];
                }
            }
            d_back = d0;
            e0 = e1;
            s0 = s1;
            w0 = w1;
            h[0] = h_on[0];
            ih[0] = ih_on[0];
        }
    }
}

// ------------------------------------------------------------------ host side

// Every element offset of the field fits 31 bits (strides may be negative).
bool offsets_fit(sil_field const& f)
{
    int64_t const lim = (int64_t(1) << 31) - 1;
    int64_t reach = 0;
    auto add = [&](int64_t stride, int64_t count) {
        if (count <= 1) return stride > -lim && stride < lim;
        if (stride > lim || stride < -lim || count > lim) return false;
        reach += (stride < 0 ? -stride : stride) * (count - 1);
        return reach < lim;
    };
    if (!add(f.comp_stride, f.ncomp)) return false;
    for (int d = 0; d < f.ndims; ++d)
        if (!add(f.stride[d], f.extent[d])) return false;
    return true;
}

template <class T, int N>
Dense<T, N> dense_args(Geometry const* geo, sil_field const& in, sil_field const& out, int64_t total)
{
    Dense<T, N> a {};
    a.in = static_cast<T const*>(in.data);
    a.out = static_cast<T*>(out.data);
    for (int d = 0; d < N; ++d) {
        a.iext[d] = static_cast<int>(in.extent[d]);
        a.istr[d] = static_cast<int>(in.stride[d]);
        a.oext[d] = static_cast<int>(out.extent[d]);
        a.ostr[d] = static_cast<int>(out.stride[d]);
        a.off[d] = static_cast<int>(out.front[d] - in.front[d]);
        if (geo != nullptr) {
            GeoView<T> const g = geo_view<T>(*geo);
            int64_t const at = in.front[d] - g.front[d] + 1;
            a.h[d] = g.h[d] + at;
            a.ih[d] = g.inv_h[d] + at;
        }
    }
    a.ics = static_cast<int>(in.comp_stride);
    a.ocs = static_cast<int>(out.comp_stride);
    a.total = static_cast<uint32_t>(total);
    return a;
}

// Dynamic shared memory a kernel may take without asking for it, so that the
// marching launches have no call that can fail before them.
constexpr size_t kPlainSmem = 48 * 1024;

// Tile height and resident CTAs: at 161x144x130 the FP64 1-form took 62.9 us
// with two CTAs of 8 rows, 53.8 with three, 61.6 with four, 58.9 with two of 12
// and 63.8 with one of 16; the other ranks and FP32 differ by less than 5 %.
constexpr int kLap3Y = 8;
template <class T, int K>
constexpr int kLap3Ctas = sizeof(T) == 8 && K == 1 ? 3 : 2;

// From how many nodes on the 3D march is taken.  1- and 2-forms: always (node
// kernel -> march, 1-form FP64: 16^3 6.4 -> 3.1 us, 64^3 20.2 -> 9.6, 161x144x130
// 143 -> 54), but for boxes whose columns the tiles cover badly (kLap3Steps).
// 0- and 3-forms read seven nodes and gain less: at similar sides once they leave
// L2 (0-form FP64: 64^3 5.9 -> 6.8, 96^3 11.9 -> 14.4, 161x144x130 30.1 -> 26.7;
// 3-form 39.1 -> 29.7); long boxes lie to either side of it (4000x7x31 14.1 -> 6.7,
// 2000x33x33 33.2 -> 45.7).
template <int K>
constexpr int64_t kLap3Min = K == 1 || K == 2 ? 1 : 2000000;

// 1- and 2-forms: the most thread steps a node (threads of the tiles times
// planes + 2 over columns times planes) at which a box of more than kLap3Small
// nodes marches; smaller ones gain from the march's shorter chain whatever the
// tiles cover.  Node kernel -> march, 1-form FP64 us, by steps: 5.0 4000x8x32 73 ->
// 48, 5.2 12x1000x12 13.9 -> 9.9, 7.3 4000x31x7 62.9 -> 57.0 (component first 62.4
// -> 85.2), 8.5 3x3x100000 24.6 -> 27.9, 11 700x700x5 164 -> 225, 65 100000x3x3 39.8
// -> 246; small: 10 16^3 6.4 -> 3.1, 24 100x9x9 6.0 -> 4.1.
constexpr int64_t kLap3Steps = 7, kLap3Small = 40000;

// The output box lies inside the input box.
template <int N, class T>
bool box_inside(Dense<T, N> const& a)
{
    for (int d = 0; d < N; ++d)
        if (a.off[d] < 0 || a.off[d] + a.oext[d] > a.iext[d]) return false;
    return true;
}

template <class T, int K>
bool launch_lap3(cudaStream_t stream, Dense<T, 3> const& a)
{
    constexpr size_t smem = sizeof(Lap3Smem<T, K, kLap3Y>);
    static_assert(smem <= kPlainSmem);
    auto const kernel = lap3_march_kernel<T, K, kLap3Y, kLap3Ctas<T, K>>;
    int const tz = (a.oext[2] + kMarchZ - 3) / (kMarchZ - 2), ty = (a.oext[1] + kLap3Y - 3) / (kLap3Y - 2);
    int64_t const columns = static_cast<int64_t>(tz) * ty;
    int const planes = run_length(columns, a.oext[0], static_cast<int64_t>(kLap3Ctas<T, K>) * multiprocessors());
    if ((K == 1 || K == 2) && a.total > kLap3Small
        && columns * (kMarchZ * kLap3Y) * (planes + 2) > kLap3Steps * a.oext[1] * a.oext[2] * planes)
        return false;
    int64_t const blocks = columns * ((a.oext[0] + planes - 1) / planes);
    if (blocks >= (int64_t(1) << 31)) return false;
    kernel<<<static_cast<unsigned>(blocks), kMarchZ * kLap3Y, smem, stream>>>(a, tz, ty, planes);
    return true;
}

// At 150x171x128 the FP64 2-form took 39.8 us with four CTAs of 8 rows, 39.1
// with three (FP32 and the other ranks 3 % slower), 48.2 with five, 45.7 with
// three of 12 rows and 47.5 with two of 16.
constexpr int kCodiff3Y = 8, kCodiff3Ctas = 4;

// Whether the 3D codifferential marches: boxes of 500,000 nodes on, below which
// too few planes are in flight (FP64, node kernel -> march: 32^3 2-form 3.2 ->
// 3.8 us, 64^3 7.7 -> 7.6, 1-form 5.7 -> 6.5; 80^3 11.5 -> 8.6 and 8.1 -> 6.9),
// whose columns the tiles cover without too many idle ones: 300x300x24 2-form
// 51.0 -> 28.0 (tiles of 1.30 times its columns), 200x9x400 11.3 -> 12.9 (1.57);
// a 1-form writes one component and gains less: 96^3 12.4 -> 13.3 (1.32),
// 110^3 15.0 -> 14.4 (1.14).
template <int K, class T>
bool codiff3_marches(Dense<T, 3> const& a)
{
    int64_t const columns = static_cast<int64_t>(a.oext[1]) * a.oext[2];
    int64_t const tz = (a.oext[2] + kMarchZ - 2) / (kMarchZ - 1), ty = (a.oext[1] + kCodiff3Y - 2) / (kCodiff3Y - 1);
    int64_t const covered = tz * (kMarchZ - 1) * ty * (kCodiff3Y - 1);
    return columns * a.oext[0] >= 500000 && covered * 4 <= columns * (K == 1 ? 5 : 6) && box_inside(a);
}

template <class T, int K>
bool launch_codiff3(cudaStream_t stream, Dense<T, 3> const& a)
{
    constexpr size_t smem = sizeof(Codiff3Smem<T, K, kCodiff3Y>);
    static_assert(smem <= kPlainSmem);
    auto const kernel = codiff3_march_kernel<T, K, kCodiff3Y, kCodiff3Ctas>;
    int const tz = (a.oext[2] + kMarchZ - 2) / (kMarchZ - 1), ty = (a.oext[1] + kCodiff3Y - 2) / (kCodiff3Y - 1);
    int64_t const columns = static_cast<int64_t>(tz) * ty;
    int const planes = run_length(columns, a.oext[0], static_cast<int64_t>(kCodiff3Ctas) * multiprocessors());
    int64_t const blocks = columns * ((a.oext[0] + planes - 1) / planes);
    if (blocks >= (int64_t(1) << 31)) return false;
    kernel<<<static_cast<unsigned>(blocks), kMarchZ * kCodiff3Y, smem, stream>>>(a, tz, ty, planes);
    return true;
}

template <class T>
bool launch_lap2(cudaStream_t stream, Dense<T, 2> const& a)
{
    int const strips = (a.oext[1] + kStripOwn - 1) / kStripOwn, groups = (strips + kStripThreads / 32 - 1) / (kStripThreads / 32);
    int const rows = run_length(groups, a.oext[0], 2 * static_cast<int64_t>(multiprocessors()));
    int64_t const blocks = static_cast<int64_t>(groups) * ((a.oext[0] + rows - 1) / rows);
    if (blocks >= (int64_t(1) << 31)) return false;
    bool const vec = a.ics == 1 && a.ocs == 1 && a.istr[1] == 2 && a.ostr[1] == 2 && a.istr[0] % 2 == 0 && a.ostr[0] % 2 == 0
                     && reinterpret_cast<uintptr_t>(a.in) % (2 * sizeof(T)) == 0
                     && reinterpret_cast<uintptr_t>(a.out) % (2 * sizeof(T)) == 0;
    auto const kernel = vec ? lap2_strip_kernel<T, true> : lap2_strip_kernel<T, false>;
    kernel<<<static_cast<unsigned>(blocks), kStripThreads, 0, stream>>>(a, strips, rows);
    return true;
}

template <int OP, class T, int N, int K = 0>
bool launch_rank(cudaStream_t stream, Geometry const* geo, int k, sil_field const& in, sil_field const& out,
                 int64_t total)
{
    if constexpr (K <= N) {
        if (k != K) return launch_rank<OP, T, N, K + 1>(stream, geo, k, in, out, total);
        if constexpr (out_comps<OP, N, K>() > 0) {
            auto const a = dense_args<T, N>(geo, in, out, total);
            if constexpr (OP == kLaplacian && N == 3)
                if (total >= kLap3Min<K> && box_inside(a) && launch_lap3<T, K>(stream, a)) return true;
            if constexpr (OP == kCodiff && N == 3)
                if (codiff3_marches<K>(a) && launch_codiff3<T, K>(stream, a)) return true;
            if constexpr (OP == kLaplacian && N == 2 && K == 1)
                if (box_inside(a) && launch_lap2<T>(stream, a)) return true;
            unsigned const blocks = static_cast<unsigned>((total + kDenseBlock - 1) / kDenseBlock);
            dense_kernel<OP, K, T, N><<<blocks, kDenseBlock, 0, stream>>>(a);
            return true;
        }
    }
    return false;
}

template <int OP, class T>
bool launch_dims(cudaStream_t stream, Geometry const* geo, int k, sil_field const& in, sil_field const& out,
                 int64_t total)
{
    switch (in.ndims) {
    case 1: return launch_rank<OP, T, 1>(stream, geo, k, in, out, total);
    case 2: return launch_rank<OP, T, 2>(stream, geo, k, in, out, total);
    case 3: return launch_rank<OP, T, 3>(stream, geo, k, in, out, total);
    default: return false;
    }
}

} // namespace

// The fields these kernels take: 1-3 lattice dims that are all form dims, and
// element offsets, node counts and box distances within 31 bits, which is what
// their 32-bit index arithmetic holds; at every size measured they were the
// faster ones (5 to 22 times on the fields above).  Everything else (spectator
// dims, four form dims, larger fields) stays with the table-driven kernels,
// which take any of it.  in and out have passed the entry point's checks.
bool dense_ok(uint32_t mask, sil_field const& in, sil_field const& out)
{
    if (in.ndims < 1 || in.ndims > 3 || mask != (1u << in.ndims) - 1) return false;
    int64_t const lim = int64_t(1) << 30;
    int64_t nodes = 1;
    for (int d = 0; d < in.ndims; ++d) {
        int64_t const off = out.front[d] - in.front[d];
        if (off <= -lim || off >= lim || in.extent[d] >= lim || out.extent[d] >= lim) return false;
        if (in.extent[d] < 1 || out.extent[d] < 1) return false;
        nodes *= out.extent[d];
        if (nodes >= (int64_t(1) << 31)) return false;
    }
    return offsets_fit(in) && offsets_fit(out);
}

// op: 0 d, 1 d^T, 2 codifferential, 3 Laplacian of a k-form; geo NULL for d
// and d^T.  Returns false, with nothing launched, for a rank without output.
bool launch_dense(cudaStream_t stream, int op, Geometry const* geo, int k, sil_field const& in, sil_field const& out)
{
    int64_t const total = node_count(out);
    bool const f64 = in.dtype == SIL_F64;
    switch (op) {
    case kD: return f64 ? launch_dims<kD, double>(stream, geo, k, in, out, total)
                        : launch_dims<kD, float>(stream, geo, k, in, out, total);
    case kDT: return f64 ? launch_dims<kDT, double>(stream, geo, k, in, out, total)
                         : launch_dims<kDT, float>(stream, geo, k, in, out, total);
    case kCodiff: return f64 ? launch_dims<kCodiff, double>(stream, geo, k, in, out, total)
                             : launch_dims<kCodiff, float>(stream, geo, k, in, out, total);
    default: return f64 ? launch_dims<kLaplacian, double>(stream, geo, k, in, out, total)
                        : launch_dims<kLaplacian, float>(stream, geo, k, in, out, total);
    }
}

} // namespace sil
