// lap2d.cu -- specialised single-pass 2D Hodge Laplacian kernels.
//
//  * 0-form (delta d): one thread per output node, 5-point stencil through
//    L1/L2 (the configuration it serves, 512^2 FP64, is L2 resident).
//  * 1-form (delta d + d delta): persistent column-strip kernel.  Input row
//    tiles of (R rows) x (128 + halo columns) x 2 components are staged into
//    shared memory by TMA (cp.async.bulk.tensor, no multicast) through an
//    S-stage mbarrier ring; each thread owns one output column and marches
//    down the rows keeping a 2-row register window, so every input element
//    leaves HBM once and every output element is written once.
//
// Both kernels evaluate exactly the same expressions, in the same order, as
// the table-driven fused kernel in dec_generic.cu, so the two agree bit for
// bit; both follow the reference composition (laplacian.hpp:27-155,
// codifferential.hpp:439-507) with the Hodge star of an orthogonal grid.
#include <cuda.h>
#include <cudaTypedefs.h>

#include <algorithm>
#include <type_traits>
#include <mutex>

#include "sil_internal.cuh"

namespace sil {

namespace {

// ------------------------------------------------------------------ 0-form

template <class T>
struct Lap0Params
{
    T const* in;
    T* out;
    int64_t nx, ny;          // input extents (x slow, y fast)
    int64_t in_row;          // input row stride (elements)
    int64_t mx, my;          // output extents
    int64_t out_row;         // output row stride
    int64_t ox, oy;          // output front relative to the input front
    T const* hx;             // padded: [p + 1]
    T const* ihx;
    T const* hy;
    T const* ihy;
};

template <class T>
__global__ void __launch_bounds__(256) lap2d_0form_kernel(Lap0Params<T> P)
{
    grid_dependency_wait();
    grid_launch_dependents();
    int64_t const jj = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x;
    int64_t const ii = blockIdx.y;
    if (jj >= P.my || ii >= P.mx) return;
    int64_t const i = ii + P.ox, j = jj + P.oy;
    auto phi = [&](int64_t p, int64_t q) {
        p = min(max(p, int64_t(0)), P.nx - 1);
        q = min(max(q, int64_t(0)), P.ny - 1);
        return __ldg(P.in + p * P.in_row + q);
    };
    // eta_x(p) = (-hx/hy) * dphi_y(p), eta_y(p) = (hy/hx) * dphi_x(p); zero outside.
    auto eta_x = [&](int64_t p, int64_t q) -> T {
        if (p < 0 || q < 0 || p >= P.nx || q >= P.ny) return T(0);
        T const d = (T(0) - phi(p, q)) + phi(p, q + 1);
        T const f = (T(-1) * __ldg(P.hx + p + 1)) * __ldg(P.ihy + q + 1);
        return f * d;
    };
    auto eta_y = [&](int64_t p, int64_t q) -> T {
        if (p < 0 || q < 0 || p >= P.nx || q >= P.ny) return T(0);
        T const d = (T(0) - phi(p, q)) + phi(p + 1, q);
        T const f = (T(1) * __ldg(P.ihx + p + 1)) * __ldg(P.hy + q + 1);
        return f * d;
    };
    T acc = T(0);
    acc = acc - eta_y(i, j);
    acc = acc + eta_x(i, j);
    acc = acc + eta_y(i - 1, j);
    acc = acc - eta_x(i, j - 1);
    T const dual_codiff = -acc;
    T const f = (T(1) * __ldg(P.ihx + i + 1)) * __ldg(P.ihy + j + 1);
    P.out[ii * P.out_row + jj] = T(-1) * (f * dual_codiff);
}

// ------------------------------------------------------------------ 1-form, TMA

constexpr int kTJ = 256;                 // output columns per strip = consumer threads
constexpr int kHalf = kTJ / 2;           // nodes per TMA box row (one half strip)
constexpr int kConsumerWarps = kTJ / 32;
constexpr int kThreads1 = kTJ + 32;      // consumers + one TMA producer warp

template <class T>
struct Lap1Traits;
template <>
struct Lap1Traits<double>
{
    using Vec = double2;
};
template <>
struct Lap1Traits<float>
{
    using Vec = float2;
};

// Pipeline shape: ROWS rows per stage, STAGES stages in the ring, MINB CTAs
// per SM the register budget is sized for.  The autotuner picks one.
//
// Stage layout in shared memory (bytes, 128-byte aligned pieces):
//   half A      ROWS rows x 128 nodes x 2 components (strip columns 0..127)
//   half B      ROWS rows x 128 nodes x 2 components (strip columns 128..255)
//   halo L      ROWS x 16 bytes: node col0-1 (FP32: the node pair col0-2, col0-1)
//   halo R      ROWS x 16 bytes: node col0+256 (FP32: the pair col0+256, col0+257)
//   factors     ROWS x (hx, 1/hx), written by the producer warp
// The 2D tensor maps view a row of the field as 2*ny contiguous elements, so
// every box row is a 2 KB (FP64) / 1 KB (FP32) contiguous run.
template <class T, int ROWS, int STAGES, int MINB>
struct Lap1Cfg
{
    using Vec = typename Lap1Traits<T>::Vec;
    static constexpr int kRows = ROWS;
    static constexpr int kStages = STAGES;
    static constexpr int kMinBlocks = MINB;
    static constexpr int kHalfBytes = ROWS * kHalf * 2 * static_cast<int>(sizeof(T));
    static constexpr int kHaloBytes = ROWS * 16;
    static constexpr int kHaloPad = (kHaloBytes + 127) / 128 * 128;
    static constexpr int kOffB = kHalfBytes;
    static constexpr int kOffL = 2 * kHalfBytes;
    static constexpr int kOffR = kOffL + kHaloPad;
    static constexpr int kOffF = kOffR + kHaloPad;
    static constexpr int kStageStride = (kOffF + ROWS * 2 * static_cast<int>(sizeof(T)) + 127) / 128 * 128;
    static constexpr int kTxBytes = 2 * kHalfBytes + 2 * kHaloBytes;
    static constexpr int kSmemBytes = STAGES * kStageStride + 128;
};

template <class T>
struct Lap1Params
{
    T* out;
    int64_t out_row;           // output row stride (elements)
    int nx, ny;                // input extents
    int mx, my;                // output extents
    int ox, oy;                // output front relative to the input front
    int strips;                // column strips of width kTJ over the output
    int band;                  // rows per band
    int64_t work;              // bands * strips * band row items, band-major: the
                               // strips of one band of rows are consecutive items
    T const* hx;               // padded spacing arrays [p + 1] (inverse pads are 0)
    T const* ihx;
    T const* hy;
    T const* ihy;
    int* error_flag;           // set when a bounded wait runs out
    int wait_tries;            // bound of each pipeline wait, in mbarrier polls
};

__device__ __forceinline__ uint32_t smem_addr(void const* p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes)
                 : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}

constexpr int kWaitTries = 1 << 22;

// Bounded wait on an mbarrier phase (at most max_tries polls; 0: the wait
// runs out at once); returns false when the bound runs out.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int max_tries = kWaitTries)
{
    uint32_t const addr = smem_addr(bar);
    for (int tries = 0; tries < max_tries; ++tries) {
        uint32_t done;
        asm volatile(
                "{\n\t.reg .pred p;\n\t"
                "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                "selp.u32 %0, 1, 0, p;\n\t}"
                : "=r"(done)
                : "r"(addr), "r"(parity)
                : "memory");
        if (done) return true;
    }
    return false;
}

__device__ __forceinline__ void tma_load_2d(void* dst, CUtensorMap const* map, uint64_t* bar, int c0, int c1)
{
    asm volatile(
            "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
            ::"r"(smem_addr(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(smem_addr(bar))
            : "memory");
}

// One strip segment of the persistent work split: strip, output rows
// [r_begin, r_end) relative to the output front (empty for the items of the
// last band that lie past the output).  The items run band by band, and
// within a band strip by strip, so the CTAs working at the same time read
// neighbouring pieces of the same rows.
struct Segment
{
    int strip, r_begin, r_end;
};

template <class T>
__device__ __forceinline__ Segment next_segment(Lap1Params<T> const& P, int64_t& item, int64_t end)
{
    Segment s;
    int64_t const blk = item / P.band;
    int const r = static_cast<int>(item - blk * P.band);
    s.strip = static_cast<int>(blk % P.strips);
    int const b = static_cast<int>(blk / P.strips);
    int64_t const len = min(end - item, static_cast<int64_t>(P.band - r));
    s.r_begin = b * P.band + r;
    s.r_end = min(s.r_begin + static_cast<int>(len), P.mx);
    item += len;
    return s;
}

template <class T, class C>
__global__ void __launch_bounds__(kThreads1, C::kMinBlocks)
lap2d_1form_tma_kernel(const __grid_constant__ CUtensorMap map_main, const __grid_constant__ CUtensorMap map_halo,
                       Lap1Params<T> P)
{
    using Vec = typename C::Vec;
    constexpr int R = C::kRows;
    constexpr int S = C::kStages;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    unsigned char* stages = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
    __shared__ __align__(8) uint64_t full[S];
    __shared__ __align__(8) uint64_t empty[S];
    __shared__ int abort_flag;

    int const tid = threadIdx.x;
    int const warp = tid / 32, lane = tid % 32;
    if (tid == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], kConsumerWarps);
        }
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
    grid_dependency_wait();
    grid_launch_dependents();

    int64_t const begin = (P.work * blockIdx.x) / gridDim.x;
    int64_t const end = (P.work * (blockIdx.x + 1)) / gridDim.x;
    // Element offset of node (., col) in the 2*ny-wide rows of the tensor maps.
    constexpr int kHaloNodes = sizeof(T) == 8 ? 1 : 2;  // nodes in a 16-byte halo box

    if (warp == kConsumerWarps) {
        // ---------------- producer warp: TMA loads + row factors
        int64_t g = 0;  // stages issued so far (all segments)
        bool ok = true;
        int64_t item = begin;
        while (item < end && ok) {
            Segment const sg = next_segment(P, item, end);
            if (sg.r_end <= sg.r_begin) continue;
            int const col0 = P.oy + sg.strip * kTJ;
            int const load_row0 = P.ox + sg.r_begin - 1;
            int const nload = sg.r_end - sg.r_begin + 2;
            int const nstages = (nload + R - 1) / R;
            for (int st = 0; st < nstages; ++st, ++g) {
                int const slot = static_cast<int>(g % S);
                uint32_t const use = static_cast<uint32_t>(g / S);
                if (use > 0) {
                    bool const got = mbar_wait(&empty[slot], (use - 1) & 1u, P.wait_tries);
                    if (!__all_sync(0xffffffffu, got) || *reinterpret_cast<volatile int*>(&abort_flag)) {
                        ok = false;
                        break;
                    }
                }
                unsigned char* stage = stages + slot * C::kStageStride;
                int const row0 = load_row0 + st * R;
                if (lane < R) {
                    int const idx = min(row0 + lane + 1, P.nx + 1);
                    T* fac = reinterpret_cast<T*>(stage + C::kOffF);
                    fac[2 * lane] = __ldg(P.hx + idx);
                    fac[2 * lane + 1] = __ldg(P.ihx + idx);
                }
                __syncwarp();
                if (lane == 0) {
                    mbar_expect_tx(&full[slot], C::kTxBytes);
                    tma_load_2d(stage, &map_main, &full[slot], 2 * col0, row0);
                    tma_load_2d(stage + C::kOffB, &map_main, &full[slot], 2 * (col0 + kHalf), row0);
                    tma_load_2d(stage + C::kOffL, &map_halo, &full[slot], 2 * (col0 - kHaloNodes), row0);
                    tma_load_2d(stage + C::kOffR, &map_halo, &full[slot], 2 * (col0 + kTJ), row0);
                }
            }
        }
        if (!ok && lane == 0) {
            abort_flag = 1;
            atomicExch(P.error_flag, 1);
            // Let the loads still in flight land (bounded) before the CTA exits.
            for (int64_t q = max(g - S, int64_t(0)); q < g; ++q)
                mbar_wait(&full[q % S], static_cast<uint32_t>(q / S) & 1u);
        }
        return;
    }

    // ---------------- consumer warps: one output column per thread
    // Neighbour addressing (in Vec units from the stage base): offset of
    // row 0 and stride between rows, for the left / own / right columns.
    constexpr int kVecPerHalfRow = kHalf;
    constexpr int kHaloStride = 16 / static_cast<int>(sizeof(Vec));
    int const half = tid / kHalf, lc = tid % kHalf;
    int const o_off = half * (C::kOffB / static_cast<int>(sizeof(Vec))) + lc;
    int m_off, m_stride, p_off, p_stride;
    if (tid == 0) {
        m_off = C::kOffL / static_cast<int>(sizeof(Vec)) + (sizeof(T) == 4 ? 1 : 0);
        m_stride = kHaloStride;
    } else if (tid == kHalf) {
        m_off = kHalf - 1;
        m_stride = kVecPerHalfRow;
    } else {
        m_off = o_off - 1;
        m_stride = kVecPerHalfRow;
    }
    if (tid == kTJ - 1) {
        p_off = C::kOffR / static_cast<int>(sizeof(Vec));
        p_stride = kHaloStride;
    } else if (tid == kHalf - 1) {
        p_off = C::kOffB / static_cast<int>(sizeof(Vec));
        p_stride = kVecPerHalfRow;
    } else {
        p_off = o_off + 1;
        p_stride = kVecPerHalfRow;
    }

    int64_t g = 0;
    int64_t item = begin;
    while (item < end) {
        Segment const sg = next_segment(P, item, end);
        if (sg.r_end <= sg.r_begin) continue;
        int const col0 = P.oy + sg.strip * kTJ;
        int const j = col0 + tid;
        int const i_first = P.ox + sg.r_begin;
        int const nload = sg.r_end - sg.r_begin + 2;
        int const nstages = (nload + R - 1) / R;

        int const jq = min(j, P.ny - 2);  // columns past the output: clamped, never stored
        T const ihy_m = __ldg(P.ihy + jq);
        T const hy_0 = __ldg(P.hy + jq + 1), ihy_0 = __ldg(P.ihy + jq + 1);
        T const hy_p = __ldg(P.hy + jq + 2), ihy_p = __ldg(P.ihy + jq + 2);
        bool const store_col = j < P.oy + P.my;

        // Window state (previous row r-1 unless noted).
        T a_m = 0, b_m = 0, a_0 = 0, b_0 = 0, a_p = 0;  // 1-form components A (x), B (y) at j-1, j, j+1
        T xy_0 = 0, xx_0 = 0, xy_p = 0, xx_p = 0;       // star of the 1-form: xi_y, xi_x at j, j+1
        T xy_p_prev = 0;                               // xi_y at row r-2, column j+1
        T s0_prev = 0, sm_prev = 0, sp_prev = 0;        // 1/(hx hy) at (r-1, j), (r-1, j-1), (r-1, j+1)
        T px0_prev = 0, qy0_prev = 0;                   // hx/hy and hy/hx at (r-1, j)
        T eta_prev = 0;                                // eta(r-2, j)
        T delta_prev = 0;                              // delta(r-1, j)
        // Rows stream from i_first - 1; output row i is complete once row i + 1
        // has arrived, so the first two streamed rows store nothing.  The eta /
        // delta values they produce are overwritten before they are used.
        int out_after = 2;
        Vec* optr = reinterpret_cast<Vec*>(P.out + static_cast<int64_t>(i_first - P.ox) * P.out_row) + (j - P.oy);
        int64_t const ostep = P.out_row / 2;  // in Vec units

        auto row_step = [&](Vec const vm, Vec const v0, Vec const vp, T const hx_r, T const ihx_r) {
            // Hodge factors at row r (zero inverse pads make every factor that
            // reaches outside the lattice vanish).
            T const px_m = hx_r * ihy_m;
            T const qy_0 = ihx_r * hy_0;
            T const px_0 = hx_r * ihy_0;
            T const qy_p = ihx_r * hy_p;
            T const px_p = hx_r * ihy_p;
            T const s_0 = ihx_r * ihy_0;
            T const s_m = ihx_r * ihy_m;
            T const s_p = ihx_r * ihy_p;
            // Star of the 1-form at row r: xi_x = -(hx/hy) B, xi_y = (hy/hx) A.
            T const nxx_m = -(px_m * vm.y);
            T const nxy_0 = qy_0 * v0.x;
            T const nxx_0 = -(px_0 * v0.y);
            T const nxy_p = qy_p * vp.x;
            T const nxx_p = -(px_p * vp.y);
            // eta = star(d w) at (r-1, j) and (r-1, j-1); chain-order sums.
            T const d0 = (((-b_0) + a_0) + v0.y) - a_p;
            T const eta_0 = s0_prev * d0;
            T const dm = (((-b_m) + a_m) + vm.y) - a_0;
            T const eta_m = sm_prev * dm;
            // delta(r, j) and delta(r-1, j+1): transposed d of xi, star, sign.
            T const acc = (((-nxy_0) + nxx_0) + xy_0) - nxx_m;
            T const delta_r = s_0 * acc;
            T const acc2 = (((-xy_p) + xx_p) + xy_p_prev) - xx_0;
            T const delta_up = sp_prev * acc2;
            if (out_after == 0) {
                // Output row r - 1: delta d (transposed d of eta, star, sign) + d delta.
                T const sx = (-eta_0) + eta_prev;
                T const sy = (-eta_0) + eta_m;
                T const ddx = -(px0_prev * sy);
                T const ddy = qy0_prev * sx;
                T const ex = (-delta_prev) + delta_r;
                T const ey = (-delta_prev) + delta_up;
                Vec o;
                o.x = ddx + ex;
                o.y = ddy + ey;
                if (store_col) __stcs(optr, o);
                optr += ostep;
            } else {
                --out_after;
            }
            eta_prev = eta_0;
            delta_prev = delta_r;
            xy_p_prev = xy_p;
            xy_0 = nxy_0;
            xx_0 = nxx_0;
            xy_p = nxy_p;
            xx_p = nxx_p;
            s0_prev = s_0;
            sm_prev = s_m;
            sp_prev = s_p;
            px0_prev = px_0;
            qy0_prev = qy_0;
            a_m = vm.x;
            b_m = vm.y;
            a_0 = v0.x;
            b_0 = v0.y;
            a_p = vp.x;
        };

        for (int st = 0; st < nstages; ++st, ++g) {
            int const slot = static_cast<int>(g % S);
            uint32_t const use = static_cast<uint32_t>(g / S);
            if (!mbar_wait(&full[slot], use & 1u, P.wait_tries)) {
                if (lane == 0) {
                    abort_flag = 1;
                    atomicExch(P.error_flag, 1);
                }
                return;
            }
            Vec const* sv = reinterpret_cast<Vec const*>(stages + slot * C::kStageStride);
            Vec const* pm = sv + m_off;
            Vec const* p0 = sv + o_off;
            Vec const* pp = sv + p_off;
            T const* fac = reinterpret_cast<T const*>(stages + slot * C::kStageStride + C::kOffF);
            int const rows_here = min(R, nload - st * R);
            if (rows_here == R) {
#pragma unroll
                for (int rr = 0; rr < R; ++rr)
                    row_step(pm[rr * m_stride], p0[rr * kVecPerHalfRow], pp[rr * p_stride], fac[2 * rr], fac[2 * rr + 1]);
            } else {
                for (int rr = 0; rr < rows_here; ++rr)
                    row_step(pm[rr * m_stride], p0[rr * kVecPerHalfRow], pp[rr * p_stride], fac[2 * rr], fac[2 * rr + 1]);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty[slot]);
        }
    }
}

// ------------------------------------------------------------------ 1-form, TMA, column pairs (FP64)
//
// The same pipeline over 512-column strips: each consumer thread owns two
// adjacent columns A = 2t, B = 2t + 1 and reads the four columns A-1..B+1 of
// a row from shared memory.  Every value the two columns have in common is
// formed once (the Hodge-factor products of columns A and B, the star of the
// 1-form at A and B, eta at A, and delta(r-1, B), which is column A's
// delta_up), so a row costs about two thirds of the single-column kernel's
// instructions per output node, and the two columns' dependency chains
// interleave.  Each shared value is the same expression, in the same order,
// as the single-column kernel evaluates it, so the outputs are bit-identical.

constexpr int kTJ2 = 512;               // output columns per strip
constexpr int kQuarter = 128;           // nodes per TMA box row (one quarter strip)

template <int ROWS, int STAGES>
struct Lap1PairCfg
{
    static constexpr int kRows = ROWS;
    static constexpr int kStages = STAGES;
    static constexpr int kQuarterBytes = ROWS * kQuarter * 16;      // FP64: 16 B per node (2 components)
    static constexpr int kHaloBytes = ROWS * 16;
    static constexpr int kHaloPad = (kHaloBytes + 127) / 128 * 128;
    static constexpr int kOffL = 4 * kQuarterBytes;
    static constexpr int kOffR = kOffL + kHaloPad;
    static constexpr int kOffF = kOffR + kHaloPad;
    static constexpr int kStageStride = (kOffF + ROWS * 16 + 127) / 128 * 128;
    static constexpr int kTxBytes = 4 * kQuarterBytes + 2 * kHaloBytes;
    static constexpr int kSmemBytes = STAGES * kStageStride + 128;
};

template <class C>
__global__ void __launch_bounds__(kThreads1, 1)
lap2d_1form_pair_kernel(const __grid_constant__ CUtensorMap map_main, const __grid_constant__ CUtensorMap map_halo,
                        Lap1Params<double> P)
{
    using Vec = double2;
    constexpr int R = C::kRows;
    constexpr int S = C::kStages;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    unsigned char* stages = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
    __shared__ __align__(8) uint64_t full[S];
    __shared__ __align__(8) uint64_t empty[S];
    __shared__ int abort_flag;

    int const tid = threadIdx.x;
    int const warp = tid / 32, lane = tid % 32;
    if (tid == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], kConsumerWarps);
        }
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
    grid_dependency_wait();
    grid_launch_dependents();

    int64_t const begin = (P.work * blockIdx.x) / gridDim.x;
    int64_t const end = (P.work * (blockIdx.x + 1)) / gridDim.x;

    if (warp == kConsumerWarps) {
        // ---------------- producer warp: TMA loads + row factors
        int64_t g = 0;
        bool ok = true;
        int64_t item = begin;
        while (item < end && ok) {
            Segment const sg = next_segment(P, item, end);
            if (sg.r_end <= sg.r_begin) continue;
            int const col0 = P.oy + sg.strip * kTJ2;
            int const load_row0 = P.ox + sg.r_begin - 1;
            int const nload = sg.r_end - sg.r_begin + 2;
            int const nstages = (nload + R - 1) / R;
            for (int st = 0; st < nstages; ++st, ++g) {
                int const slot = static_cast<int>(g % S);
                uint32_t const use = static_cast<uint32_t>(g / S);
                if (use > 0) {
                    bool const got = mbar_wait(&empty[slot], (use - 1) & 1u, P.wait_tries);
                    if (!__all_sync(0xffffffffu, got) || *reinterpret_cast<volatile int*>(&abort_flag)) {
                        ok = false;
                        break;
                    }
                }
                unsigned char* stage = stages + slot * C::kStageStride;
                int const row0 = load_row0 + st * R;
                if (lane < R) {
                    int const idx = min(row0 + lane + 1, P.nx + 1);
                    double* fac = reinterpret_cast<double*>(stage + C::kOffF);
                    fac[2 * lane] = __ldg(P.hx + idx);
                    fac[2 * lane + 1] = __ldg(P.ihx + idx);
                }
                __syncwarp();
                if (lane == 0) {
                    mbar_expect_tx(&full[slot], C::kTxBytes);
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        tma_load_2d(stage + q * C::kQuarterBytes, &map_main, &full[slot], 2 * (col0 + q * kQuarter), row0);
                    tma_load_2d(stage + C::kOffL, &map_halo, &full[slot], 2 * (col0 - 1), row0);
                    tma_load_2d(stage + C::kOffR, &map_halo, &full[slot], 2 * (col0 + kTJ2), row0);
                }
            }
        }
        if (!ok && lane == 0) {
            abort_flag = 1;
            atomicExch(P.error_flag, 1);
            for (int64_t q = max(g - S, int64_t(0)); q < g; ++q)
                mbar_wait(&full[q % S], static_cast<uint32_t>(q / S) & 1u);
        }
        return;
    }

    // ---------------- consumer warps: columns A = 2 tid, B = 2 tid + 1 of the strip
    constexpr int kQV = C::kQuarterBytes / 16;  // Vecs per quarter block
    int const q = tid / 64, c0 = 2 * (tid % 64);
    int const oA = q * kQV + c0;
    int m_off, m_stride, p_off, p_stride;
    if (c0 > 0) {
        m_off = oA - 1;
        m_stride = kQuarter;
    } else if (q > 0) {
        m_off = (q - 1) * kQV + kQuarter - 1;
        m_stride = kQuarter;
    } else {
        m_off = C::kOffL / 16;
        m_stride = 1;
    }
    if (c0 + 1 < kQuarter - 1) {
        p_off = oA + 2;
        p_stride = kQuarter;
    } else if (q < 3) {
        p_off = (q + 1) * kQV;
        p_stride = kQuarter;
    } else {
        p_off = C::kOffR / 16;
        p_stride = 1;
    }

    int64_t g = 0;
    int64_t item = begin;
    while (item < end) {
        Segment const sg = next_segment(P, item, end);
        if (sg.r_end <= sg.r_begin) continue;
        int const col0 = P.oy + sg.strip * kTJ2;
        int const jA = col0 + 2 * tid;
        int const i_first = P.ox + sg.r_begin;
        int const nload = sg.r_end - sg.r_begin + 2;
        int const nstages = (nload + R - 1) / R;

        // Column constants from A's clamped index: columns past the output
        // are never stored, and a stored column sees exactly the factors the
        // single-column kernel gives it.
        int const jq = min(jA, P.ny - 2);
        double const ihy_M = __ldg(P.ihy + jq);
        double const hy_A = __ldg(P.hy + jq + 1), ihy_A = __ldg(P.ihy + jq + 1);
        double const hy_B = __ldg(P.hy + jq + 2), ihy_B = __ldg(P.ihy + jq + 2);
        double const hy_P = __ldg(P.hy + jq + 3), ihy_P = __ldg(P.ihy + jq + 3);
        bool const storeA = jA < P.oy + P.my;
        bool const storeB = jA + 1 < P.oy + P.my;

        double a_M = 0, b_M = 0, a_A = 0, b_A = 0, a_B = 0, b_B = 0, a_P = 0;   // components at row r-1
        double xy_A = 0, xx_A = 0, xy_B = 0, xx_B = 0, xy_P = 0, xx_P = 0;     // star at row r-1
        double xyB_prev = 0, xyP_prev = 0;                                    // xi_y at row r-2
        double sA_prev = 0, sM_prev = 0, sB_prev = 0, sP_prev = 0;            // 1/(hx hy) at row r-1
        double pxA_prev = 0, qyA_prev = 0, pxB_prev = 0, qyB_prev = 0;        // hx/hy, hy/hx at row r-1
        double etaA_prev = 0, etaB_prev = 0;                                  // eta at row r-2
        double dA_prev = 0, dB_prev = 0;                                      // delta at row r-1
        int out_after = 2;
        Vec* optr = reinterpret_cast<Vec*>(P.out + static_cast<int64_t>(i_first - P.ox) * P.out_row) + (jA - P.oy);
        int64_t const ostep = P.out_row / 2;

        auto row_step = [&](Vec const vM, Vec const vA, Vec const vB, Vec const vP, double const hx_r,
                            double const ihx_r) {
            double const px_M = hx_r * ihy_M;
            double const qy_A = ihx_r * hy_A;
            double const px_A = hx_r * ihy_A;
            double const qy_B = ihx_r * hy_B;
            double const px_B = hx_r * ihy_B;
            double const s_A = ihx_r * ihy_A;
            double const s_M = ihx_r * ihy_M;
            double const s_B = ihx_r * ihy_B;
            double const qy_P = ihx_r * hy_P;
            double const px_P = hx_r * ihy_P;
            double const s_P = ihx_r * ihy_P;
            double const nxx_M = -(px_M * vM.y);
            double const nxy_A = qy_A * vA.x;
            double const nxx_A = -(px_A * vA.y);
            double const nxy_B = qy_B * vB.x;
            double const nxx_B = -(px_B * vB.y);
            double const nxy_P = qy_P * vP.x;
            double const nxx_P = -(px_P * vP.y);
            // eta at row r-1: columns A, A-1 (A's eta_m) and B (B's eta_m is eta at A)
            double const d0A = (((-b_A) + a_A) + vA.y) - a_B;
            double const etaA = sA_prev * d0A;
            double const dmA = (((-b_M) + a_M) + vM.y) - a_A;
            double const etaM = sM_prev * dmA;
            double const d0B = (((-b_B) + a_B) + vB.y) - a_P;
            double const etaB = sB_prev * d0B;
            // delta(r, A), delta(r, B), and delta(r-1, B+1) (B's delta_up); A's
            // delta_up is delta(r-1, B) = dB_prev
            double const accA = (((-nxy_A) + nxx_A) + xy_A) - nxx_M;
            double const dA = s_A * accA;
            double const accB = (((-nxy_B) + nxx_B) + xy_B) - nxx_A;
            double const dB = s_B * accB;
            double const acc2B = (((-xy_P) + xx_P) + xyP_prev) - xx_B;
            double const dupB = sP_prev * acc2B;
            if (out_after == 0) {
                Vec o;
                {
                    double const sx = (-etaA) + etaA_prev;
                    double const sy = (-etaA) + etaM;
                    double const ddx = -(pxA_prev * sy);
                    double const ddy = qyA_prev * sx;
                    double const ex = (-dA_prev) + dA;
                    double const ey = (-dA_prev) + dB_prev;
                    o.x = ddx + ex;
                    o.y = ddy + ey;
                    if (storeA) __stcs(optr, o);
                }
                {
                    double const sx = (-etaB) + etaB_prev;
                    double const sy = (-etaB) + etaA;
                    double const ddx = -(pxB_prev * sy);
                    double const ddy = qyB_prev * sx;
                    double const ex = (-dB_prev) + dB;
                    double const ey = (-dB_prev) + dupB;
                    o.x = ddx + ex;
                    o.y = ddy + ey;
                    if (storeB) __stcs(optr + 1, o);
                }
                optr += ostep;
            } else {
                --out_after;
            }
            etaA_prev = etaA;
            etaB_prev = etaB;
            dA_prev = dA;
            dB_prev = dB;
            xyB_prev = xy_B;
            xyP_prev = xy_P;
            xy_A = nxy_A;
            xx_A = nxx_A;
            xy_B = nxy_B;
            xx_B = nxx_B;
            xy_P = nxy_P;
            xx_P = nxx_P;
            sA_prev = s_A;
            sM_prev = s_M;
            sB_prev = s_B;
            sP_prev = s_P;
            pxA_prev = px_A;
            qyA_prev = qy_A;
            pxB_prev = px_B;
            qyB_prev = qy_B;
            a_M = vM.x;
            b_M = vM.y;
            a_A = vA.x;
            b_A = vA.y;
            a_B = vB.x;
            b_B = vB.y;
            a_P = vP.x;
        };

        for (int st = 0; st < nstages; ++st, ++g) {
            int const slot = static_cast<int>(g % S);
            uint32_t const use = static_cast<uint32_t>(g / S);
            if (!mbar_wait(&full[slot], use & 1u, P.wait_tries)) {
                if (lane == 0) {
                    abort_flag = 1;
                    atomicExch(P.error_flag, 1);
                }
                return;
            }
            Vec const* sv = reinterpret_cast<Vec const*>(stages + slot * C::kStageStride);
            Vec const* pm = sv + m_off;
            Vec const* pa = sv + oA;
            Vec const* pp = sv + p_off;
            double const* fac = reinterpret_cast<double const*>(stages + slot * C::kStageStride + C::kOffF);
            int const rows_here = min(R, nload - st * R);
            if (rows_here == R) {
#pragma unroll
                for (int rr = 0; rr < R; ++rr)
                    row_step(pm[rr * m_stride], pa[rr * kQuarter], pa[rr * kQuarter + 1], pp[rr * p_stride],
                             fac[2 * rr], fac[2 * rr + 1]);
            } else {
                for (int rr = 0; rr < rows_here; ++rr)
                    row_step(pm[rr * m_stride], pa[rr * kQuarter], pa[rr * kQuarter + 1], pp[rr * p_stride],
                             fac[2 * rr], fac[2 * rr + 1]);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty[slot]);
        }
    }
}

} // namespace

// ------------------------------------------------------------------ host side

namespace {

PFN_cuTensorMapEncodeTiled_v12000 encode_fn()
{
    static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess
            && q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
    });
    return fn;
}

int sm_count()
{
    static int n = 0;
    if (n == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
        if (n <= 0) n = 1;
    }
    return n;
}

} // namespace

// Fields the specialised 2D kernels accept: both form dims, contiguous DDC
// layout (component fastest, then y, then x), output box inside the input.  The
// scalar one has a row of blocks per output row, so no more rows than a grid has
// along y.
bool lap2d_layout_ok(sil_field const& in, sil_field const& out, int ncomp)
{
    if (in.ndims != 2 || out.ndims != 2 || in.ncomp != ncomp || out.ncomp != ncomp) return false;
    if (in.dtype != out.dtype) return false;
    if (ncomp == 2 && (in.comp_stride != 1 || out.comp_stride != 1)) return false;
    if (in.stride[1] != ncomp || out.stride[1] != ncomp) return false;
    if (in.stride[0] != ncomp * in.extent[1]) return false;
    if (out.stride[0] < ncomp * out.extent[1]) return false;
    for (int d = 0; d < 2; ++d) {
        if (out.front[d] < in.front[d]) return false;
        if (out.front[d] + out.extent[d] > in.front[d] + in.extent[d]) return false;
    }
    if (ncomp == 1 && out.extent[0] > 65535) return false;
    return in.extent[0] >= 2 && in.extent[1] >= 2;
}

// Block widths the 0-form kernel's tuner chooses from (threads along y).
constexpr int kLap0Widths[3] = {64, 128, 256};
constexpr int kLap0Variants = 3;

sil_status launch_lap2d_0form(cudaStream_t stream, Geometry const& geo, sil_field const& in, sil_field const& out,
                              int variant)
{
    int64_t const mx = out.extent[0], my = out.extent[1];
    if (mx == 0 || my == 0) return SIL_OK;
    int const bx = kLap0Widths[(variant >= 0 && variant < kLap0Variants) ? variant : kLap0Variants - 1];
    dim3 const block(bx);
    dim3 const grid(static_cast<unsigned>((my + bx - 1) / bx), static_cast<unsigned>(mx));
    int64_t const gx = in.front[0] - geo.front[0], gy = in.front[1] - geo.front[1];
    if (in.dtype == SIL_F64) {
        Lap0Params<double> P {static_cast<double const*>(in.data), static_cast<double*>(out.data), in.extent[0],
                              in.extent[1], in.stride[0], mx, my, out.stride[0], out.front[0] - in.front[0],
                              out.front[1] - in.front[1], geo.h[0] + gx, geo.inv_h[0] + gx, geo.h[1] + gy,
                              geo.inv_h[1] + gy};
        SIL_CUDA_CHECK(launch_pdl(lap2d_0form_kernel<double>, grid, block, 0, stream, P));
    } else {
        Lap0Params<float> P {static_cast<float const*>(in.data), static_cast<float*>(out.data), in.extent[0],
                             in.extent[1], in.stride[0], mx, my, out.stride[0], out.front[0] - in.front[0],
                             out.front[1] - in.front[1], geo.h32[0] + gx, geo.inv_h32[0] + gx, geo.h32[1] + gy,
                             geo.inv_h32[1] + gy};
        SIL_CUDA_CHECK(launch_pdl(lap2d_0form_kernel<float>, grid, block, 0, stream, P));
    }
    SIL_CUDA_CHECK(cudaGetLastError());
    return SIL_OK;
}

sil_status launch_lap2d_0form(cudaStream_t stream, Geometry const& geo, sil_field const& in, sil_field const& out)
{
    return launch_lap2d_0form(stream, geo, in, out, kLap0Variants - 1);
}

// Time every block width on the caller's fields (two warm-up and twenty
// timed launches each, the field stays in L2 as in use) and return the
// fastest.  Runs on `stream` and synchronises it.
sil_status autotune_lap2d_0form(cudaStream_t stream, Geometry const& geo, sil_field const& in, sil_field const& out,
                                int* best_variant)
{
    cudaEvent_t e0, e1;
    SIL_CUDA_CHECK(cudaEventCreate(&e0));
    SIL_CUDA_CHECK(cudaEventCreate(&e1));
    float best = 1e30f;
    int best_v = kLap0Variants - 1;
    sil_status st = SIL_OK;
    for (int v = 0; v < kLap0Variants && st == SIL_OK; ++v) {
        for (int i = 0; i < 2 && st == SIL_OK; ++i) st = launch_lap2d_0form(stream, geo, in, out, v);
        cudaEventRecord(e0, stream);
        for (int i = 0; i < 20 && st == SIL_OK; ++i) st = launch_lap2d_0form(stream, geo, in, out, v);
        cudaEventRecord(e1, stream);
        cudaError_t const err = cudaEventSynchronize(e1);
        if (err != cudaSuccess) {
            st = cuda_fail(err, "autotune");
            break;
        }
        float ms = 0.f;
        cudaEventElapsedTime(&ms, e0, e1);
        if (ms < best) {
            best = ms;
            best_v = v;
        }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    *best_variant = best_v;
    return st;
}

// The TMA 1-form kernel additionally needs the output box to stay one node
// away from the input's upper edges (no clamped samples), 16-byte aligned
// rows, int-sized extents, and for FP32 an even y extent and even y offset.
bool lap2d_1form_tma_ok(sil_field const& in, sil_field const& out)
{
    if (!lap2d_layout_ok(in, out, 2)) return false;
    int64_t const ox = out.front[0] - in.front[0], oy = out.front[1] - in.front[1];
    if (ox + out.extent[0] > in.extent[0] - 1 || oy + out.extent[1] > in.extent[1] - 1) return false;
    if (in.extent[0] > (1 << 30) || in.extent[1] > (1 << 30)) return false;
    size_t const es = in.dtype == SIL_F64 ? 8 : 4;
    if (reinterpret_cast<uintptr_t>(in.data) % 16 != 0) return false;
    if (reinterpret_cast<uintptr_t>(out.data) % (2 * es) != 0) return false;
    if ((out.stride[0] * es) % (2 * es) != 0) return false;
    if (in.dtype == SIL_F32 && (in.extent[1] % 2 != 0 || oy % 2 != 0)) return false;
    return encode_fn() != nullptr;
}

namespace {

template <class T, class C>
int lap1_occupancy()
{
    static int blocks = -1;
    if (blocks < 0) {
        cudaFuncSetAttribute(lap2d_1form_tma_kernel<T, C>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes);
        int b = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, lap2d_1form_tma_kernel<T, C>, kThreads1, C::kSmemBytes);
        blocks = b > 0 ? b : 0;
    }
    return blocks;
}

template <class T, class C>
sil_status launch_variant(cudaStream_t stream, Geometry const& geo, sil_field const& in, sil_field const& out,
                          int* error_flag, int ctas_per_sm, int wait_tries)
{
    auto encode = encode_fn();
    if (encode == nullptr) return fail(SIL_ERR_UNSUPPORTED, "cuTensorMapEncodeTiled is unavailable");
    int64_t const mx = out.extent[0], my = out.extent[1];
    uint64_t const nx = in.extent[0], ny = in.extent[1];
    constexpr bool f64 = sizeof(T) == 8;
    // Rows of 2*ny contiguous elements; the main boxes cover half a strip
    // (128 nodes), the halo boxes one 16-byte slot (1 node FP64, 2 nodes FP32).
    cuuint64_t dims[2] = {2 * ny, nx};
    cuuint64_t strides[1] = {2 * ny * sizeof(T)};
    cuuint32_t box_main[2] = {2 * kHalf, static_cast<cuuint32_t>(C::kRows)};
    cuuint32_t box_halo[2] = {16 / sizeof(T), static_cast<cuuint32_t>(C::kRows)};
    cuuint32_t estr[2] = {1, 1};
    auto const dt = f64 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32;
    CUtensorMap map_main, map_halo;
    CUresult res = encode(&map_main, dt, 2, in.data, dims, strides, box_main, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                          CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (res == CUDA_SUCCESS)
        res = encode(&map_halo, dt, 2, in.data, dims, strides, box_halo, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (res != CUDA_SUCCESS) return fail(SIL_ERR_CUDA, "cuTensorMapEncodeTiled failed");
    int const occ = lap1_occupancy<T, C>();
    if (occ < 1) return fail(SIL_ERR_UNSUPPORTED, "1-form Laplacian variant does not fit on an SM");
    int const strips = static_cast<int>((my + kTJ - 1) / kTJ);
    int const per_sm = ctas_per_sm > 0 ? std::min(ctas_per_sm, occ) : occ;
    int64_t ctas = std::min<int64_t>(static_cast<int64_t>(strips) * mx, static_cast<int64_t>(sm_count()) * per_sm);
    if (ctas < 1) ctas = 1;
    int const bands = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(mx, ctas / strips)));
    int const band = static_cast<int>((mx + bands - 1) / bands);
    int64_t const work = static_cast<int64_t>(bands) * strips * band;
    int64_t const gx = in.front[0] - geo.front[0], gy = in.front[1] - geo.front[1];
    T const* const* gh = reinterpret_cast<T const* const*>(f64 ? (void const*)geo.h : (void const*)geo.h32);
    T const* const* gih = reinterpret_cast<T const* const*>(f64 ? (void const*)geo.inv_h : (void const*)geo.inv_h32);
    Lap1Params<T> P {static_cast<T*>(out.data), out.stride[0], static_cast<int>(nx), static_cast<int>(ny),
                     static_cast<int>(mx), static_cast<int>(my), static_cast<int>(out.front[0] - in.front[0]),
                     static_cast<int>(out.front[1] - in.front[1]), strips, band, work, gh[0] + gx, gih[0] + gx,
                     gh[1] + gy, gih[1] + gy, error_flag, wait_tries};
    SIL_CUDA_CHECK(launch_pdl(lap2d_1form_tma_kernel<T, C>, static_cast<unsigned>(ctas), kThreads1, C::kSmemBytes, stream,
                              map_main, map_halo, P));
    return SIL_OK;
}

template <class C>
int lap1_pair_occupancy()
{
    static int blocks = -1;
    if (blocks < 0) {
        cudaFuncSetAttribute(lap2d_1form_pair_kernel<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, C::kSmemBytes);
        int b = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, lap2d_1form_pair_kernel<C>, kThreads1, C::kSmemBytes);
        blocks = b > 0 ? b : 0;
    }
    return blocks;
}

// The column-pair kernel (FP64): 512-column strips, the same tensor maps as
// the single-column kernel with this shape's rows per box.
template <class C>
sil_status launch_pair_variant(cudaStream_t stream, Geometry const& geo, sil_field const& in, sil_field const& out,
                               int* error_flag, int wait_tries)
{
    auto encode = encode_fn();
    if (encode == nullptr) return fail(SIL_ERR_UNSUPPORTED, "cuTensorMapEncodeTiled is unavailable");
    int64_t const mx = out.extent[0], my = out.extent[1];
    uint64_t const nx = in.extent[0], ny = in.extent[1];
    cuuint64_t dims[2] = {2 * ny, nx};
    cuuint64_t strides[1] = {2 * ny * sizeof(double)};
    cuuint32_t box_main[2] = {2 * kQuarter, static_cast<cuuint32_t>(C::kRows)};
    cuuint32_t box_halo[2] = {2, static_cast<cuuint32_t>(C::kRows)};
    cuuint32_t estr[2] = {1, 1};
    CUtensorMap map_main, map_halo;
    CUresult res = encode(&map_main, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 2, in.data, dims, strides, box_main, estr,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (res == CUDA_SUCCESS)
        res = encode(&map_halo, CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 2, in.data, dims, strides, box_halo, estr,
                     CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (res != CUDA_SUCCESS) return fail(SIL_ERR_CUDA, "cuTensorMapEncodeTiled failed");
    int const occ = lap1_pair_occupancy<C>();
    if (occ < 1) return fail(SIL_ERR_UNSUPPORTED, "1-form Laplacian pair variant does not fit on an SM");
    int const strips = static_cast<int>((my + kTJ2 - 1) / kTJ2);
    int64_t ctas = std::min<int64_t>(static_cast<int64_t>(strips) * mx, static_cast<int64_t>(sm_count()) * occ);
    if (ctas < 1) ctas = 1;
    int const bands = static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(mx, ctas / strips)));
    int const band = static_cast<int>((mx + bands - 1) / bands);
    int64_t const work = static_cast<int64_t>(bands) * strips * band;
    int64_t const gx = in.front[0] - geo.front[0], gy = in.front[1] - geo.front[1];
    Lap1Params<double> P {static_cast<double*>(out.data), out.stride[0], static_cast<int>(nx), static_cast<int>(ny),
                          static_cast<int>(mx), static_cast<int>(my), static_cast<int>(out.front[0] - in.front[0]),
                          static_cast<int>(out.front[1] - in.front[1]), strips, band, work, geo.h[0] + gx,
                          geo.inv_h[0] + gx, geo.h[1] + gy, geo.inv_h[1] + gy, error_flag, wait_tries};
    SIL_CUDA_CHECK(launch_pdl(lap2d_1form_pair_kernel<C>, static_cast<unsigned>(ctas), kThreads1, C::kSmemBytes, stream,
                              map_main, map_halo, P));
    return SIL_OK;
}

// Candidate pipeline shapes (rows per stage, stages, CTAs per SM sized for).
template <class T>
struct Lap1Variants;
template <>
struct Lap1Variants<double>
{
    using V0 = Lap1Cfg<double, 4, 4, 2>;
    using V1 = Lap1Cfg<double, 4, 6, 2>;
    using V2 = Lap1Cfg<double, 8, 3, 2>;
    using V3 = Lap1Cfg<double, 8, 6, 1>;
    using V4 = Lap1Cfg<double, 2, 8, 2>;
    using V5 = Lap1Cfg<double, 16, 3, 1>;
};
template <>
struct Lap1Variants<float>
{
    using V0 = Lap1Cfg<float, 4, 4, 3>;
    using V1 = Lap1Cfg<float, 4, 8, 2>;
    using V2 = Lap1Cfg<float, 8, 4, 2>;
    using V3 = Lap1Cfg<float, 8, 8, 1>;
    using V4 = Lap1Cfg<float, 2, 8, 3>;
    using V5 = Lap1Cfg<float, 16, 4, 1>;
};

constexpr int kLap1Variants = 6;      // single-column shapes (FP64 and FP32)
constexpr int kLap1PairVariants = 3;  // column-pair shapes (FP64 only), indices 6..8

int lap1_variant_count(bool f64)
{
    return kLap1Variants + (f64 ? kLap1PairVariants : 0);
}

template <class T>
sil_status launch_by_index(int v, cudaStream_t stream, Geometry const& geo, sil_field const& in, sil_field const& out,
                           int* error_flag, int ctas_per_sm, int wait_tries)
{
    using V = Lap1Variants<T>;
    switch (v) {
    case 0: return launch_variant<T, typename V::V0>(stream, geo, in, out, error_flag, ctas_per_sm, wait_tries);
    case 1: return launch_variant<T, typename V::V1>(stream, geo, in, out, error_flag, ctas_per_sm, wait_tries);
    case 2: return launch_variant<T, typename V::V2>(stream, geo, in, out, error_flag, ctas_per_sm, wait_tries);
    case 3: return launch_variant<T, typename V::V3>(stream, geo, in, out, error_flag, ctas_per_sm, wait_tries);
    case 4: return launch_variant<T, typename V::V4>(stream, geo, in, out, error_flag, ctas_per_sm, wait_tries);
    case 6:
        if constexpr (std::is_same_v<T, double>)
            return launch_pair_variant<Lap1PairCfg<8, 3>>(stream, geo, in, out, error_flag, wait_tries);
        else
            return launch_variant<T, typename V::V0>(stream, geo, in, out, error_flag, ctas_per_sm, wait_tries);
    case 7:
        if constexpr (std::is_same_v<T, double>)
            return launch_pair_variant<Lap1PairCfg<4, 6>>(stream, geo, in, out, error_flag, wait_tries);
        else
            return launch_variant<T, typename V::V0>(stream, geo, in, out, error_flag, ctas_per_sm, wait_tries);
    case 8:
        if constexpr (std::is_same_v<T, double>)
            return launch_pair_variant<Lap1PairCfg<2, 12>>(stream, geo, in, out, error_flag, wait_tries);
        else
            return launch_variant<T, typename V::V0>(stream, geo, in, out, error_flag, ctas_per_sm, wait_tries);
    default: return launch_variant<T, typename V::V5>(stream, geo, in, out, error_flag, ctas_per_sm, wait_tries);
    }
}

} // namespace

int lap2d_1form_variants()
{
    return kLap1Variants + kLap1PairVariants;
}

// Launch pipeline variant `variant` (0 = default) of the TMA 1-form kernel;
// wait_tries bounds each pipeline wait (< 0: the default bound).
sil_status launch_lap2d_1form_tma(cudaStream_t stream, Geometry const& geo, sil_field const& in, sil_field const& out,
                                  int* error_flag, int variant, int wait_tries)
{
    if (out.extent[0] == 0 || out.extent[1] == 0) return SIL_OK;
    if (variant < 0 || variant >= lap1_variant_count(in.dtype == SIL_F64)) variant = 0;
    int const tries = wait_tries < 0 ? kWaitTries : wait_tries;
    if (in.dtype == SIL_F64) return launch_by_index<double>(variant, stream, geo, in, out, error_flag, 0, tries);
    return launch_by_index<float>(variant, stream, geo, in, out, error_flag, 0, tries);
}

sil_status launch_lap2d_1form_tma(cudaStream_t stream, Geometry const& geo, sil_field const& in, sil_field const& out,
                                  int* error_flag, int variant)
{
    return launch_lap2d_1form_tma(stream, geo, in, out, error_flag, variant, -1);
}

// Time every variant on the caller's fields (two warm-up and three timed
// launches each) and return the fastest.  Runs on `stream` and synchronises it.
sil_status autotune_lap2d_1form(cudaStream_t stream, Geometry const& geo, sil_field const& in, sil_field const& out,
                                int* error_flag, int* best_variant, float* best_ms)
{
    // Shapes are timed as CUDA graphs of back-to-back launches (the way
    // repeated runs reach the GPU, the programmatic launch overlap included).
    // Screening: every shape that fits, a graph of 10 launches replayed in a
    // warm-up and two timed rounds that interleave the shapes.  Final: the
    // two fastest, a graph of 40 launches each, alternated over three timed
    // rounds after a warm-up; a shape's time is its fastest round.
    int const nv = lap1_variant_count(in.dtype == SIL_F64);
    std::vector<cudaGraphExec_t> exec(nv, nullptr);
    std::vector<float> t(nv, 1e30f);
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    cudaStream_t cs = nullptr;
    sil_status st = SIL_OK;
    auto drop_graphs = [&]() {
        for (cudaGraphExec_t& g : exec)
            if (g != nullptr) {
                cudaGraphExecDestroy(g);
                g = nullptr;
            }
    };
    auto cleanup = [&]() {
        drop_graphs();
        if (e0 != nullptr) cudaEventDestroy(e0);
        if (e1 != nullptr) cudaEventDestroy(e1);
        if (cs != nullptr) cudaStreamDestroy(cs);
    };
    if (cudaEventCreate(&e0) != cudaSuccess || cudaEventCreate(&e1) != cudaSuccess
        || cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking) != cudaSuccess) {
        cleanup();
        return fail(SIL_ERR_CUDA, "autotune: event or stream creation failed");
    }
    auto capture = [&](int v, int launches) -> sil_status {
        cudaGraph_t graph = nullptr;
        sil_status cst = SIL_OK;
        cudaError_t err = cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal);
        for (int i = 0; i < launches && err == cudaSuccess && cst == SIL_OK; ++i)
            cst = launch_lap2d_1form_tma(cs, geo, in, out, error_flag, v);
        cudaError_t const err2 = cudaStreamEndCapture(cs, &graph);
        if (err == cudaSuccess) err = err2;
        if (err == cudaSuccess && cst == SIL_OK) err = cudaGraphInstantiate(&exec[v], graph, 0);
        if (graph != nullptr) cudaGraphDestroy(graph);
        if (cst != SIL_OK) return cst;
        return err == cudaSuccess ? SIL_OK : cuda_fail(err, "autotune graph");
    };
    auto rounds = [&](std::vector<int> const& vs, int launches, int timed) -> sil_status {
        for (int round = 0; round <= timed; ++round) {
            for (int v : vs) {
                cudaEventRecord(e0, stream);
                cudaError_t err = cudaGraphLaunch(exec[v], stream);
                cudaEventRecord(e1, stream);
                if (err == cudaSuccess) err = cudaEventSynchronize(e1);
                if (err != cudaSuccess) return cuda_fail(err, "autotune");
                float ms = 0.f;
                cudaEventElapsedTime(&ms, e0, e1);
                if (round > 0) t[v] = std::min(t[v], ms / launches);  // round 0 warms up
            }
        }
        return SIL_OK;
    };
    std::vector<int> fit;
    for (int v = 0; v < nv && st == SIL_OK; ++v) {
        sil_status const probe = launch_lap2d_1form_tma(stream, geo, in, out, error_flag, v);
        if (probe == SIL_ERR_UNSUPPORTED) continue;  // does not fit: skip
        if (probe != SIL_OK) {
            st = probe;
            break;
        }
        st = capture(v, 10);
        if (st == SIL_OK) fit.push_back(v);
    }
    if (st == SIL_OK) st = rounds(fit, 10, 2);
    if (st == SIL_OK && fit.size() > 1) {
        std::vector<int> top = fit;
        std::sort(top.begin(), top.end(), [&](int a, int b) { return t[a] < t[b]; });
        top.resize(2);
        drop_graphs();
        for (int v : top) {
            t[v] = 1e30f;
            if (st == SIL_OK) st = capture(v, 40);
        }
        for (int v : fit)
            if (v != top[0] && v != top[1]) t[v] = 1e30f;
        if (st == SIL_OK) st = rounds(top, 40, 3);
    }
    cleanup();
    int best_v = fit.empty() ? 0 : fit[0];
    for (int v : fit)
        if (t[v] < t[best_v]) best_v = v;
    *best_variant = best_v;
    *best_ms = t[best_v];
    return st;
}

} // namespace sil
