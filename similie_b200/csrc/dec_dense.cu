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
// sides).
#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include <type_traits>

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

template <int OP, class T, int N, int K = 0>
bool launch_rank(cudaStream_t stream, Geometry const* geo, int k, sil_field const& in, sil_field const& out,
                 int64_t total)
{
    if constexpr (K <= N) {
        if (k != K) return launch_rank<OP, T, N, K + 1>(stream, geo, k, in, out, total);
        if constexpr (out_comps<OP, N, K>() > 0) {
            auto const a = dense_args<T, N>(geo, in, out, total);
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
