// precond.cu -- kernels and host driver of the learned multilevel
// convolutional preconditioner (network layout in precond_net.cuh).
//
// Activation storage: one buffer per level holding every image of the batch
// that reaches that level; an image of h x w pixels is stored padded to
// (h+2) x (w+2) pixels with a zero border, 32 channels fastest (BF16,
// 64 bytes per pixel), so a 3x3 tap is a flat pixel offset.  Gradients of
// activations are FP32 in the same layout.
//
// 32->32 convolutions run on the tensor cores as implicit GEMMs: a CTA owns
// 128 consecutive flat pixels (M = 128), N = 32 output channels, K = 9 taps
// x 32 input channels.  The three 130-pixel halo rows of the tile are staged
// once in shared memory in the canonical no-swizzle UMMA layout (16-byte
// channel chunks, pixels at 16-byte stride), so each of the 9 taps is an
// operand descriptor at a different start address; 18 tcgen05.mma
// (128x32x16, BF16 in, FP32 accumulate in TMEM) per tile, one commit, the
// epilogue reads TMEM with tcgen05.ld and applies bias / ReLU / border.
// The weight gradient runs on the tensor cores too (M = 4 taps x 32 input
// channels from an im2col tile, N = 32, K = pixels, MN-major operands),
// accumulating in TMEM over all tiles of a persistent CTA.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>
#include <vector>

#include "mag_ops.cuh"
#include "precond_net.cuh"
#include "sil_internal.cuh"
#include "sm100.cuh"

namespace sil {
namespace nn {

using bf16 = __nv_bfloat16;
using namespace sil::sm100;

constexpr int kTilePx = 128;
constexpr int kHalo = kTilePx + 2;
constexpr int kChunks = kCh / 8;                 // 16-byte chunks per pixel
constexpr int kKChunks = kTaps * kChunks;        // 36
constexpr int kWgradParts = kBigW + kCh;         // per-CTA partial: weights + bias
constexpr uint32_t kIdescFwd = idesc_bf16_f32(128, 32, false, false);
constexpr uint32_t kIdescWgrad = idesc_bf16_f32(128, 32, true, true);

struct Img
{
    int32_t h, w;     // interior pixels
    int64_t offset;   // pixel offset of the padded image in its level buffer
};

// Images of one launch: output level and, per image, the other level the
// input mode reads (POOL: the finer level; UPADD: the coarser level).
struct Table
{
    int nimg;
    int32_t tile_base[kMaxImages + 1];
    Img img[kMaxImages];
    Img aux[kMaxImages];
    int32_t sample[kMaxImages];   // batch sample of each image
    int const* active;            // per batch sample: 0 = skip its images (NULL: all run)
    int64_t px_base[kMaxImages + 1];  // prefix of padded pixels: the images as one flat range
};

// An image whose sample is switched off is neither read nor written.
__device__ __forceinline__ bool image_active(Table const& t, int im)
{
    return t.active == nullptr || __ldg(t.active + t.sample[im]) != 0;
}

// Convolution inputs: kPlain the level's own tensor; kUpAdd skip + nearest
// upsampled coarse tensor (two operands summed by the tensor core); kMasked a
// FP32 gradient masked by ReLU activity (data gradients).
enum InMode { kPlain = 0, kUpAdd, kMasked, kModes };

__device__ __forceinline__ void unpack8(uint4 u, float* f)
{
    __nv_bfloat162 const* h = reinterpret_cast<__nv_bfloat162 const*>(&u);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float2 const t = __bfloat1622float2(h[i]);
        f[2 * i] = t.x;
        f[2 * i + 1] = t.y;
    }
}

__device__ __forceinline__ uint4 pack8(float const* f)
{
    uint4 u;
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&u);
#pragma unroll
    for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
    return u;
}

// Two FP32 fused multiply-adds in one instruction, each rounded as __fmaf_rn.
struct Float2x
{
    uint64_t v;
};
__device__ __forceinline__ Float2x pair2(float lo, float hi)
{
    Float2x r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ float2 split2(Float2x p)
{
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(p.v));
    return r;
}
__device__ __forceinline__ Float2x fma2(Float2x a, Float2x b, Float2x c)
{
    Float2x r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}

__device__ __forceinline__ int find_image(Table const& t, int tile)
{
    int lo = 0, hi = t.nimg - 1;
    while (lo < hi) {
        int const mid = (lo + hi + 1) / 2;
        if (t.tile_base[mid] <= tile) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Work of a launch is counted in units (tiles, pixels, wrapper items) per
// image; only the units of active images are handed out.  scan_active
// forms, in shared memory, the exclusive prefix pre[0..n] over the n <= 64
// images of count(k) (0 for an inactive image): warp 0 scans two images per
// lane.  Every thread of the block must call it; it ends with a barrier.
static_assert(kMaxImages <= 64, "scan_active covers 64 images");
template <class C>
__device__ __forceinline__ void scan_active(int n, C const& count, int64_t* pre)
{
    if (threadIdx.x < 32) {
        int const lane = threadIdx.x;
        int64_t const a = 2 * lane < n ? count(2 * lane) : 0;
        int64_t const b = 2 * lane + 1 < n ? count(2 * lane + 1) : 0;
        int64_t v = a + b;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            int64_t const y = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o) v += y;
        }
        int64_t const excl = v - a - b;
        if (2 * lane < n) pre[2 * lane] = excl;
        if (2 * lane + 1 < n) pre[2 * lane + 1] = excl + a;
        if (lane == 31) pre[n] = v;
    }
    __syncthreads();
}

// Image of active unit u (u < pre[n]): the largest k with pre[k] <= u.  An
// inactive image has pre[k] == pre[k + 1], so the search never stops on one.
__device__ __forceinline__ int find_unit(int64_t const* pre, int n, int64_t u)
{
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        int const mid = (lo + hi + 1) / 2;
        if (pre[mid] <= u) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// Walk of a compacted range of `total` = pre[n] * per elements: each block
// takes one contiguous slice (a multiple of blockDim.x long), each thread
// every blockDim.x-th element of it, and the image index advances as the
// walk crosses image ends (zero-length inactive images are passed over), so
// an element costs one compare beyond f(k, q), q the element's index within
// image k.  No barrier may sit inside f.
template <class F>
__device__ __forceinline__ void walk_range(int64_t const* pre, int n, int per, F const& f)
{
    int64_t const B = blockDim.x, G = gridDim.x;
    int64_t const total = pre[n] * per;
    int64_t const slice = ((total + G - 1) / G + B - 1) / B * B;
    int64_t e = static_cast<int64_t>(blockIdx.x) * slice + threadIdx.x;
    int64_t const stop = min(total, static_cast<int64_t>(blockIdx.x + 1) * slice);
    if (e >= stop) return;
    int k = find_unit(pre, n, e / per);
    int64_t base = pre[k] * per, end = pre[k + 1] * per;
    for (; e < stop; e += B) {
        while (e >= end) {
            ++k;
            base = end;
            end = pre[k + 1] * per;
        }
        f(k, static_cast<int>(e - base));
    }
}

// Elementwise kernels: the padded pixels of the table's active images, `per`
// elements per pixel, as one compacted range; f(im, q) for element q of
// image im (q < npx(im) * per).  The cost follows the active pixels,
// whatever the number of inactive images.
template <class F>
__device__ __forceinline__ void walk_active(Table const& t, int64_t* pre, int per, F const& f)
{
    scan_active(
        t.nimg, [&](int k) { return image_active(t, k) ? t.px_base[k + 1] - t.px_base[k] : int64_t(0); }, pre);
    walk_range(pre, t.nimg, per, f);
}

// Chunk c (eight channels) of the FP32 gradient gin masked by ReLU activity, at
// padded flat pixel g of an image: zero outside the image and on its border.
// 32-bit pixel arithmetic (images below 2^31 pixels).
__device__ __forceinline__ uint4 masked_chunk(Img const& o, int g, int c, bf16 const* act, float const* gin)
{
    int const P = o.w + 2;
    uint4 const zero = make_uint4(0u, 0u, 0u, 0u);
    if (g < 0 || g >= P * (o.h + 2)) return zero;
    int const y = g / P, x = g - y * P;
    if (y == 0 || x == 0 || y > o.h || x > o.w) return zero;
    float4 const* gp = reinterpret_cast<float4 const*>(gin + (o.offset + g) * kCh) + 2 * c;
    float4 const a = __ldg(gp), b = __ldg(gp + 1);
    float av[8];
    unpack8(__ldg(reinterpret_cast<uint4 const*>(act) + (o.offset + g) * kChunks + c), av);
    float const gv[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    float f[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] = av[i] > 0.0f ? gv[i] : 0.0f;
    return pack8(f);
}

// Stage the three 130-pixel rows of the masked gradient around the tile
// starting at flat pixel `start` into smem (layout [chunk][row][pixel], 16 bytes
// per entry).  Four neighbouring lanes form a pixel's chunks, so a warp reads
// runs of whole pixels.
__device__ __forceinline__ void stage_halo_masked(uint4* halo, Img const& o, int start, bf16 const* act, float const* gin)
{
    int const P = o.w + 2, c = threadIdx.x & 3;
#pragma unroll 4
    for (int q = threadIdx.x >> 2; q < 3 * kHalo; q += 32) {
        int const r = q / kHalo, j = q - r * kHalo;
        halo[(c * 3 + r) * kHalo + j] = masked_chunk(o, start + (r - 1) * P - 1 + j, c, act, gin);
    }
}

__device__ __forceinline__ void cp_async16(uint4* dst, void const* src, bool valid)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src),
                 "r"(valid ? 16 : 0)
                 : "memory");
}

__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_group1() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }

// The level's own tensor.  Four neighbouring lanes copy the four chunks of a
// pixel, so a warp's copy reads 512 contiguous bytes and walks the row by
// constant distances; only a row that leaves the image is checked per pixel.
__device__ __forceinline__ void stage_halo_plain(uint4* halo, Table const& t, int im, int start, int P, bf16 const* src)
{
    Img const o = t.img[im];
    int const npx = P * (o.h + 2);
    int const c = threadIdx.x & 3, j0 = threadIdx.x >> 2;
    uint4 const* base = reinterpret_cast<uint4 const*>(src) + o.offset * kChunks + c;
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        int const g0 = start + (r - 1) * P - 1;
        uint4* dst = &halo[(c * 3 + r) * kHalo + j0];
        uint4 const* p = base + static_cast<int64_t>(g0 + j0) * kChunks;
        bool const whole = g0 >= 0 && g0 + kHalo <= npx;
#pragma unroll
        for (int q = 0; q < (kHalo + 31) / 32; ++q) {
            if (32 * q + 31 >= kHalo && j0 + 32 * q >= kHalo) continue;
            int const g = g0 + j0 + 32 * q;
            bool const valid = whole || (g >= 0 && g < npx);
            cp_async16(dst + 32 * q, valid ? p + 32 * q * kChunks : base, valid);
        }
    }
}

// The nearest-upsampled coarse tensor gathered to this level; pixels outside
// the image and on its border are zero-filled.
__device__ __forceinline__ void stage_halo_up(uint4* halo, Table const& t, int im, int start, int P, bf16 const* src)
{
    Img const o = t.img[im];
    int const npx = P * (o.h + 2);
    Img const ci = t.aux[im];
    uint4 const* base = reinterpret_cast<uint4 const*>(src);
    // Image coordinates of each halo row's first pixel (floor division, so
    // the pixel before the image is row -1); within a row they advance by
    // adding, wrapping at the row pitch P.
    int y0[3], x0[3];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        int const g0 = start + (r - 1) * P - 1;
        int const y = g0 >= 0 ? g0 / P : -1;
        y0[r] = y;
        x0[r] = g0 - y * P;
    }
    for (int i = threadIdx.x; i < 3 * kHalo; i += blockDim.x) {
        int const r = i / kHalo, j = i - r * kHalo;
        int const g = start + (r - 1) * P - 1 + j;
        bool valid = g >= 0 && g < npx;
        int64_t px = 0;
        if (valid) {
            int y = r == 0 ? y0[0] : (r == 1 ? y0[1] : y0[2]);
            int x = (r == 0 ? x0[0] : (r == 1 ? x0[1] : x0[2])) + j;
            while (x >= P) {
                x -= P;
                ++y;
            }
            valid = !(y == 0 || x == 0 || y > o.h || x > o.w);
            px = ci.offset + static_cast<int64_t>((y - 1) / 2 + 1) * (ci.w + 2) + ((x - 1) / 2 + 1);
        }
        uint4 const* p = valid ? base + px * kChunks : base;
#pragma unroll
        for (int c = 0; c < kChunks; ++c) cp_async16(&halo[(c * 3 + r) * kHalo + j], p + c, valid);
    }
}

// The kernels of an apply and of a gradient's backward pass follow one another
// by programmatic dependent launch: a kernel's CTAs may take their places, and do
// what needs no predecessor (the convolutions their weights, TMEM and barriers),
// while the previous kernel's last CTAs run.  after_previous comes before
// anything the previous kernel wrote is read and before anything is written, in
// every CTA, and lets the next kernel start only from there: so when a kernel
// starts, every kernel before its predecessor has finished and two at most are
// under way.  The pointers to what the predecessor wrote pass through the wait,
// so no load by them can be moved ahead of it.  B200: an apply of 36 launches,
// eight samples of 256^2 .. 1024^2, 552 -> 468 us; a gradient of eight 256^2
// samples, about 120 launches, 984 -> 836 us; a learned solve of five problems
// 149 -> 139 ms.
template <class... P>
__device__ __forceinline__ void after_previous(P const*&... read)
{
    asm volatile("griddepcontrol.wait;" ::: "memory");
    (([](P const*& p) { asm volatile("" : "+l"(p)::"memory"); })(read), ...);
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Shared memory of the convolution kernel.  The second halo (used by kUpAdd
// only) comes last, so the other modes launch with the shorter block and fit
// more CTAs per multiprocessor.
struct ConvSmem
{
    uint4 w[kKChunks * kCh];              // B operand: [K chunk][output channel], 18432 B
    float4 wout[kCh][3];                  // output-convolution weights [input channel][tap, 12 with padding]
    uint64_t bar[2];
    uint32_t tmem;
    int abort;
    int64_t pre[kMaxImages + 1];          // prefix of the active images' tiles
    uint4 halo[2][kChunks * 3 * kHalo];   // A operand sources: [chunk][halo row][halo pixel], 2 x 24960 B
};

// Where a convolution's results go: bias / ReLU applied, out (BF16), out_f32
// (with accumulate) and out_taps as conv3x3_kernel describes them.
struct ConvOut
{
    float const* bias;
    int relu;
    bf16* out;
    float* out_f32;
    int accumulate;
    float* out_taps;
    int64_t taps_stride;
};

// Epilogue of one 128-pixel tile from its accumulator (a pixel per thread).
__device__ __forceinline__ void conv_epilogue(ConvOut const& w, float const (&bias_r)[32], float4 const (*wout)[3],
                                              uint32_t tmem, Img const& o, int start)
{
    int const warp = threadIdx.x >> 5, lane = threadIdx.x & 31, P = o.w + 2;
    float acc[32];
    tmem_ld32(tmem + (static_cast<uint32_t>(warp * 32) << 16), acc);
    int const g = start + warp * 32 + lane;
    if (g < P * (o.h + 1)) {
        int const x = g % P;
        bool const border = x == 0 || x == P - 1;
        if (border) {
#pragma unroll
            for (int i = 0; i < 32; ++i) acc[i] = 0.0f;
        } else {
            if (w.bias != nullptr) {
#pragma unroll
                for (int i = 0; i < 32; ++i) acc[i] = acc[i] + bias_r[i];
            }
            if (w.relu) {
#pragma unroll
                for (int i = 0; i < 32; ++i) acc[i] = fmaxf(acc[i], 0.0f);
            }
        }
        int64_t const px = o.offset + g;
        if (w.out_f32 != nullptr) {
            float4* dst = reinterpret_cast<float4*>(w.out_f32 + px * kCh);
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                float4 v = make_float4(acc[4 * q], acc[4 * q + 1], acc[4 * q + 2], acc[4 * q + 3]);
                if (w.accumulate) {
                    float4 const o4 = dst[q];
                    v.x = v.x + o4.x;
                    v.y = v.y + o4.y;
                    v.z = v.z + o4.z;
                    v.w = v.w + o4.w;
                }
                dst[q] = v;
            }
        }
        if (w.out != nullptr || w.out_taps != nullptr) {
            uint4 packed[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) packed[q] = pack8(acc + 8 * q);
            if (w.out != nullptr) {
                uint4* dst = reinterpret_cast<uint4*>(w.out + px * kCh);
#pragma unroll
                for (int q = 0; q < 4; ++q) dst[q] = packed[q];
            }
            if (w.out_taps != nullptr) {
                // partials of the output convolution from the BF16-rounded activations
                float f[32];
#pragma unroll
                for (int q = 0; q < 4; ++q) unpack8(packed[q], f + 8 * q);
                // nine accumulators side by side, eight of them in pairs; each
                // tap still sums its 32 channels in order from zero
                Float2x a2[4];
                float a[kTaps];
#pragma unroll
                for (int k = 0; k < 4; ++k) a2[k] = pair2(0.0f, 0.0f);
                a[8] = 0.0f;
#pragma unroll
                for (int ci = 0; ci < 32; ++ci) {
                    float4 const w0 = wout[ci][0], w1 = wout[ci][1];
                    Float2x const v = pair2(f[ci], f[ci]);
                    a2[0] = fma2(pair2(w0.x, w0.y), v, a2[0]);
                    a2[1] = fma2(pair2(w0.z, w0.w), v, a2[1]);
                    a2[2] = fma2(pair2(w1.x, w1.y), v, a2[2]);
                    a2[3] = fma2(pair2(w1.z, w1.w), v, a2[3]);
                    a[8] = __fmaf_rn(wout[ci][2].x, f[ci], a[8]);
                }
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    float2 const q = split2(a2[k]);
                    a[2 * k] = q.x;
                    a[2 * k + 1] = q.y;
                }
#pragma unroll
                for (int tap = 0; tap < kTaps; ++tap) w.out_taps[tap * w.taps_stride + px] = a[tap];
            }
        }
    }
}

// The 18 MMAs of one operand, issued by one thread: descriptors differ from the
// first tap's by constant distances in their address field (16-byte units), so
// each costs two adds.
__device__ __forceinline__ void issue_taps(uint32_t tmem, uint32_t halo, uint64_t b0, bool accumulate)
{
    uint64_t const a0 = umma_desc(halo, 3 * kHalo * 16, 128);
#pragma unroll
    for (int tap = 0; tap < kTaps; ++tap) {
#pragma unroll
        for (int h = 0; h < 2; ++h)
            umma_bf16(tmem, a0 + ((2 * h * 3 + tap / 3) * kHalo + tap % 3), b0 + (tap * kChunks + 2 * h) * kCh, kIdescFwd,
                      accumulate || tap > 0 || h > 0 ? 1u : 0u);
    }
}

// What both convolution kernels do before their first tile: weights to shared
// memory, TMEM columns, the barriers.
__device__ __forceinline__ void conv_setup(ConvSmem& s, bf16 const* wt, float const* wout, uint32_t columns)
{
    int const tid = threadIdx.x;
#pragma unroll
    for (int i = 0; i < kKChunks * kCh / 128; ++i) s.w[tid + i * 128] = __ldg(reinterpret_cast<uint4 const*>(wt) + tid + i * 128);
    if (wout != nullptr)
        for (int i = tid; i < kCh * 12; i += 128) {
            int const ci = i / 12, tap = i - ci * 12;
            reinterpret_cast<float*>(s.wout[ci])[tap] = tap < kTaps ? wout[tap * kCh + ci] : 0.0f;
        }
    if (tid < 32) tmem_alloc(&s.tmem, columns);
    if (tid == 0) {
        mbar_init(&s.bar[0], 1);
        mbar_init(&s.bar[1], 1);
        s.abort = 0;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
}

__device__ __forceinline__ void conv_teardown(ConvSmem& s, int* error_flag, uint32_t columns)
{
    cp_async_wait_all();  // no copy may still target this CTA's shared memory at exit
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (s.abort && threadIdx.x == 0) atomicExch(error_flag, 1);
    if (threadIdx.x < 32) tmem_dealloc(s.tmem, columns);
}

// out = act(conv3x3(in) + bias) of a level's own tensor, for the interior pixels
// of every active image of the table (border pixels are written as zero; the
// forms of output are ConvOut's).  Two halo buffers and two accumulators keep
// one tile ahead: while a tile's epilogue runs, the next tile's MMAs run and
// the copies of the one after it are on their way, with one barrier a tile.
// Bound by latency still, with three CTAs of four warps on a multiprocessor.
// B200, the 32 -> 1 folding decoder of 1 M pixels: 101 us with the MMAs waited
// for before each epilogue, here 82.
__global__ void __launch_bounds__(128) conv3x3_plain_kernel(const __grid_constant__ Table t, bf16 const* in, bf16 const* wt,
                                                            ConvOut const dst, float const* wout, int* error_flag)
{
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    ConvSmem& s = *reinterpret_cast<ConvSmem*>(smem_raw);
    int const tid = threadIdx.x;
    scan_active(
        t.nimg, [&](int k) { return image_active(t, k) ? int64_t(t.tile_base[k + 1] - t.tile_base[k]) : int64_t(0); },
        s.pre);
    // a CTA without an active tile leaves before staging weights or taking TMEM
    int const nact = static_cast<int>(s.pre[t.nimg]), G = static_cast<int>(gridDim.x);
    if (static_cast<int>(blockIdx.x) >= nact) {
        after_previous(in);
        return;
    }
    // active tiles handed out round-robin
    struct Place
    {
        int im, start;
    };
    auto place_of = [&](int a) -> Place {
        int const k = find_unit(s.pre, t.nimg, a);
        return {k, t.img[k].w + 2 + (a - static_cast<int>(s.pre[k])) * kTilePx};
    };
    auto stage = [&](Place const& p, int buf) {
        stage_halo_plain(s.halo[buf], t, p.im, p.start, t.img[p.im].w + 2, in);
        cp_async_commit();
    };
    conv_setup(s, wt, dst.out_taps != nullptr ? wout : nullptr, 64);
    after_previous(in);
    Place now = place_of(blockIdx.x), next {};
    stage(now, 0);
    int a = blockIdx.x;
    if (a + G < nact) {
        next = place_of(a + G);
        stage(next, 1);
    }
    uint32_t const tmem = s.tmem;
    uint64_t const b0 = umma_desc(smem_u32(s.w), kCh * 16, 128);
    float bias_r[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) bias_r[i] = dst.bias != nullptr ? __ldg(dst.bias + i) : 0.0f;
    if (a + G < nact) cp_async_wait_group1();
    else cp_async_wait_all();
    fence_async_smem();
    __syncthreads();
    if (tid == 0) {
        tc_fence_after();
        issue_taps(tmem, smem_u32(s.halo[0]), b0, false);
        umma_commit(&s.bar[0]);
    }
    uint32_t phase = 0;   // bit b: parity of barrier b's next completion
    bool lost = false;
    for (int buf = 0; a < nact; a += G, buf ^= 1) {
        bool const more = a + G < nact;
        if (more) {
            // the next tile's copies have landed: its MMAs go to the other accumulator,
            // whose previous tile every warp has read by this barrier
            cp_async_wait_all();
            fence_async_smem();
            if (__syncthreads_or(lost)) break;
            if (tid == 0) {
                tc_fence_after();
                issue_taps(tmem + (buf ^ 1) * 32, smem_u32(s.halo[buf ^ 1]), b0, false);
                umma_commit(&s.bar[buf ^ 1]);
            }
            __syncwarp();
        }
        bool const done = __all_sync(0xffffffffu, mbar_wait(&s.bar[buf], (phase >> buf) & 1u));
        phase ^= 1u << buf;
        if (!done) {
            lost = true;
            s.abort = 1;
            continue;
        }
        Place after {};
        if (a + 2 * G < nact) {
            after = place_of(a + 2 * G);
            stage(after, buf);   // this tile's MMAs have read the buffer
        }
        tc_fence_after();
        conv_epilogue(dst, bias_r, s.wout, tmem + buf * 32, t.img[now.im], now.start);
        tc_fence_before();
        now = next;
        next = after;
    }
    conv_teardown(s, error_flag, 64);
}

// The other inputs of a convolution (training): kUpAdd, skip + nearest-upsampled
// coarse tensor as two operands summed in the accumulator, and kMasked, an FP32
// gradient masked by activity; one tile at a time.
__global__ void __launch_bounds__(128, 4) conv3x3_kernel(const __grid_constant__ Table t, int mode, bf16 const* in,
                                                      bf16 const* in2, float const* gin, bf16 const* wt,
                                                      ConvOut const dst, int* error_flag)
{
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    ConvSmem& s = *reinterpret_cast<ConvSmem*>(smem_raw);
    int const tid = threadIdx.x;
    conv_setup(s, wt, nullptr, 32);
    after_previous(in, in2, gin);
    uint32_t const tmem = s.tmem;
    uint32_t const halo_addr[2] = {smem_u32(s.halo[0]), smem_u32(s.halo[1])};
    uint64_t const b0 = umma_desc(smem_u32(s.w), kCh * 16, 128);
    float bias_r[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) bias_r[i] = dst.bias != nullptr ? __ldg(dst.bias + i) : 0.0f;
    uint32_t phase = 0;
    for (int tile = blockIdx.x; tile < t.tile_base[t.nimg]; tile += gridDim.x) {
        int const im = find_image(t, tile);
        Img const o = t.img[im];
        int const P = o.w + 2;
        int const start = P + (tile - t.tile_base[im]) * kTilePx;
        if (mode == kUpAdd) {
            stage_halo_plain(s.halo[0], t, im, start, P, in);
            stage_halo_up(s.halo[1], t, im, start, P, in2);
            cp_async_wait_all();
        } else {
            stage_halo_masked(s.halo[0], o, start, in2, gin);
        }
        fence_async_smem();
        __syncthreads();
        if (tid == 0) {
            tc_fence_after();
            issue_taps(tmem, halo_addr[0], b0, false);
            if (mode == kUpAdd) issue_taps(tmem, halo_addr[1], b0, true);
            umma_commit(&s.bar[0]);
        }
        __syncwarp();
        bool const done = mbar_wait(&s.bar[0], phase);
        phase ^= 1u;
        if (!done) s.abort = 1;
        __syncthreads();
        if (s.abort) break;
        tc_fence_after();
        conv_epilogue(dst, bias_r, s.wout, tmem, o, start);
        tc_fence_before();
        __syncthreads();
    }
    conv_teardown(s, error_flag, 32);
}

// Output convolution from the tap partials: out[p] = b + sum_tap taps[tap][p + tap] (zero border).
__global__ void out_gather_kernel(const __grid_constant__ Table t, float const* taps, int64_t taps_stride,
                                  float const* params, float* out)
{
    __shared__ int64_t pre[kMaxImages + 1];
    after_previous(taps);
    float const bias = params[kOffOut + kOutW];
    walk_active(t, pre, 1, [&](int im, int g) {
        Img const o = t.img[im];
        int const P = o.w + 2;
        int const y = g / P, x = g - y * P;
        float a = 0.0f;
        if (!(y == 0 || x == 0 || y > o.h || x > o.w)) {
            a = bias;
            int64_t const base = o.offset + g;
#pragma unroll
            for (int tap = 0; tap < kTaps; ++tap)
                a = a + taps[tap * taps_stride + base + (tap / 3 - 1) * P + (tap % 3 - 1)];
        }
        out[o.offset + g] = a;
    });
}

// Coarse tensor = 2x2 average of the finer level (t.img coarse, t.aux fine),
// BF16.  A thread per 16-byte chunk of a pixel, so a warp's loads and stores
// are runs of whole pixels (a thread per pixel put its lanes 128 bytes apart:
// 30 us at 1 M pixels, this one 15).
__global__ void pool_kernel(const __grid_constant__ Table t, bf16 const* fine, bf16* coarse)
{
    __shared__ int64_t pre[kMaxImages + 1];
    after_previous(fine);
    walk_active(t, pre, kChunks, [&](int im, int q) {
        Img const o = t.img[im], fi = t.aux[im];
        int const g = q / kChunks, c = q % kChunks, P = o.w + 2;
        int const y = g / P, x = g - y * P;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (!(y == 0 || x == 0 || y > o.h || x > o.w)) {
            int const Pf = fi.w + 2;
            uint4 const* src = reinterpret_cast<uint4 const*>(fine)
                               + (fi.offset + static_cast<int64_t>(2 * y - 1) * Pf + (2 * x - 1)) * kChunks + c;
            uint4 const raw[4] = {__ldg(src), __ldg(src + kChunks), __ldg(src + Pf * kChunks), __ldg(src + (Pf + 1) * kChunks)};
            float f[8], a[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) f[i] = 0.0f;
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                unpack8(raw[k], a);
#pragma unroll
                for (int i = 0; i < 8; ++i) f[i] = f[i] + a[i];
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) f[i] = f[i] * 0.25f;
            v = pack8(f);
        }
        reinterpret_cast<uint4*>(coarse)[o.offset * kChunks + q] = v;
    });
}

// Shared memory of the weight-gradient kernel.  The im2col tile is followed
// by the other buffers so that the third M tile (taps 8..11, of which only
// tap 8 exists) reads in-bounds shared memory for the missing taps.
struct WgradSmem
{
    uint4 col[kKChunks * kTilePx];     // A operand: [K-row chunk (tap, ci/8)][pixel], 73728 B
    uint4 dz[kChunks * kTilePx];       // B operand: [output-channel chunk][pixel], 8192 B
    uint4 halo[kChunks * 3 * kHalo];   // 24960 B
    uint64_t bar;
    uint32_t tmem;
    int abort;
};
static_assert(sizeof(uint4) * (kKChunks * kTilePx + kChunks * kTilePx + kChunks * 3 * kHalo)
                      >= sizeof(uint4) * 48 * kTilePx,
              "the third M tile must stay inside the shared-memory block");

// Per-CTA partial weight and bias gradients of one 32->32 convolution:
// dW[co][tap][ci] = sum_p dz[p][co] * in[p + tap][ci], db[co] = sum_p dz[p][co]
// with dz = dy * (y > 0).  The halo of the next pass or tile is copied while a
// tile's MMAs run, and all four warps share the bias sums; bound by the latency
// of a tile's phases and the im2col copy through shared memory.  B200, the
// twelve launches of a gradient of eight 256^2 samples: 194 -> 154 us against
// staging each operand pixel by pixel and one warp summing the bias.
__global__ void __launch_bounds__(128) wgrad_kernel(const __grid_constant__ Table t, int mode, bf16 const* in,
                                                    bf16 const* in2, float const* dy, bf16 const* y, float* part,
                                                    int* error_flag)
{
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    WgradSmem& s = *reinterpret_cast<WgradSmem*>(smem_raw);
    int const tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (warp == 0) tmem_alloc(&s.tmem, 128);
    if (tid == 0) {
        mbar_init(&s.bar, 1);
        s.abort = 0;
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    after_previous(in, in2, dy, y);
    uint32_t const tmem = s.tmem;
    uint64_t const a0 = umma_desc(smem_u32(s.col), 128, kTilePx * 16), b0 = umma_desc(smem_u32(s.dz), 128, kTilePx * 16);
    uint32_t phase = 0;
    float db = 0.0f;  // bias gradient of channel lane over this warp's quarter of every tile
    bool any = false;
    int const ntiles = t.tile_base[t.nimg];
    // kUpAdd: the two summands of the input in two passes (skip, then the
    // upsampled coarse tensor), both accumulated into TMEM.
    int const npass = mode == kUpAdd ? 2 : 1;
    auto stage = [&](int tile, int pass) {
        if (tile >= ntiles) return;
        int const im = find_image(t, tile), P = t.img[im].w + 2, start = P + (tile - t.tile_base[im]) * kTilePx;
        if (pass == 0) stage_halo_plain(s.halo, t, im, start, P, in);
        else stage_halo_up(s.halo, t, im, start, P, in2);
    };
    stage(blockIdx.x, 0);
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        int const im = find_image(t, tile);
        Img const o = t.img[im];
        int const P = o.w + 2, start = P + (tile - t.tile_base[im]) * kTilePx;
#pragma unroll
        for (int q = 0; q < kChunks; ++q) {
            int const m = tid / kChunks + q * 32, g = start + m, c = tid % kChunks;
            s.dz[c * kTilePx + m] = masked_chunk(o, g < P * (o.h + 1) ? g : -1, c, y, dy);
        }
        for (int pass = 0; pass < npass; ++pass) {
            cp_async_wait_all();
            __syncthreads();
#pragma unroll
            for (int kc = 0; kc < kKChunks; ++kc)
                s.col[kc * kTilePx + tid] = s.halo[(kc % kChunks * 3 + kc / kChunks / 3) * kHalo + tid + kc / kChunks % 3];
            if (pass == 0) {
                bf16 const* dz = reinterpret_cast<bf16 const*>(s.dz) + lane / 8 * kTilePx * 8 + lane % 8;
#pragma unroll 8
                for (int m = warp * 32; m < warp * 32 + 32; ++m) db = db + __bfloat162float(dz[m * 8]);
            }
            fence_async_smem();
            __syncthreads();
            if (tid == 0) {
                tc_fence_after();
#pragma unroll
                for (int mt = 0; mt < 3; ++mt) {
#pragma unroll
                    for (int kk = 0; kk < kTilePx / 16; ++kk)
                        umma_bf16(tmem + mt * 32, a0 + (16 * mt * kTilePx + kk * 16), b0 + kk * 16, kIdescWgrad,
                                  (any || kk > 0) ? 1u : 0u);
                }
                umma_commit(&s.bar);
            }
            any = true;
            __syncwarp();
            // every thread has read the halo: the next pass's or tile's takes its place
            if (pass + 1 < npass) stage(tile, pass + 1);
            else stage(tile + static_cast<int>(gridDim.x), 0);
            bool const done = mbar_wait(&s.bar, phase);
            phase ^= 1u;
            if (!done) s.abort = 1;
            __syncthreads();
            if (s.abort) break;
            tc_fence_before();
            __syncthreads();
        }
        if (s.abort) break;
    }
    cp_async_wait_all();  // no copy may still target this CTA's shared memory at exit
    __shared__ float dbs[4][kCh];
    dbs[warp][lane] = db;
    __syncthreads();
    float* dst = part + static_cast<int64_t>(blockIdx.x) * kWgradParts;
    if (!s.abort) {
        tc_fence_after();
        for (int mt = 0; mt < 3; ++mt) {
            float acc[32];
            tmem_ld32(tmem + (static_cast<uint32_t>(warp * 32) << 16) + mt * 32, acc);
            int const tap = 4 * mt + warp;
            if (tap < kTaps) {
                for (int co = 0; co < kCh; ++co) dst[co * (kTaps * kCh) + tap * kCh + lane] = any ? acc[co] : 0.0f;
            }
        }
        if (tid < kCh) dst[kBigW + tid] = dbs[0][tid] + dbs[1][tid] + dbs[2][tid] + dbs[3][tid];
    } else if (tid == 0) {
        atomicExch(error_flag, 1);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    if (warp == 0) tmem_dealloc(tmem, 128);
}

// grad[i] += sum over parts p of part[p][i], 32 entries per block: each of
// the eight warps sums a contiguous eighth of the parts in order, warp 0 adds
// the eight sums in order (a fixed order for a given number of parts).  One
// thread per entry summing all parts in series took 10.7 us a call at eight
// 256^2 samples, this 6.1.
__global__ void __launch_bounds__(256) reduce_parts_kernel(float const* part, int nparts, int n, float* grad)
{
    __shared__ float red[8][32];
    after_previous(part);
    int const warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int const i = blockIdx.x * 32 + lane;
    int const per = (nparts + 7) / 8, p1 = min(nparts, (warp + 1) * per);
    float sacc = 0.0f;
    if (i < n) {
#pragma unroll 8
        for (int p = warp * per; p < p1; ++p) sacc = sacc + part[static_cast<int64_t>(p) * n + i];
    }
    red[warp][lane] = sacc;
    __syncthreads();
    if (warp != 0 || i >= n) return;
    float total = 0.0f;
#pragma unroll
    for (int w = 0; w < 8; ++w) total = total + red[w][lane];
    grad[i] = grad[i] + total;
}

// BF16 weights of the 32->32 convolutions in the order the convolution holds
// them in shared memory, [K chunk][output channel][8 channels] with K =
// (tap, input channel), so a CTA copies them straight: forward, and for the
// data gradient transposed and flipped (K = (8 - tap, co), output ci).
__global__ void convert_weights_kernel(float const* params, bf16* wf, bf16* wt)
{
    int const i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= kNumBig * kBigW) return;
    int const j = i / kBigW, r = i % kBigW;
    int const co = r / (kTaps * kCh), tap = (r / kCh) % kTaps, ci = r % kCh;
    bf16 const v = __float2bfloat16_rn(params[kOffBig + j * kBigParams + r]);
    auto at = [](int out, int k) { return (k / 8 * kCh + out) * 8 + k % 8; };
    wf[j * kBigW + at(co, tap * kCh + ci)] = v;
    wt[j * kBigW + at(ci, (kTaps - 1 - tap) * kCh + co)] = v;
}

// ------------------------------------------------------------------ thin layers (CUDA cores)

// Input convolution 2 -> 32 (+ bias, ReLU) from the FP32 2-channel feature
// image; weights staged in shared memory.  B200, 1 M pixels: 53 us with two
// pixels of all channels per thread (its stores 128 bytes apart), here 45 with
// two multiply-adds an instruction.
constexpr int kIncRun = 4;
__global__ void __launch_bounds__(256) inc_forward_kernel(const __grid_constant__ Table t, float const* feat,
                                                          float const* params, bf16* out)
{
    // weights transposed to [input k][output channel], four channels per float4
    __shared__ float4 w4[kTaps * 2][kCh / 4];
    __shared__ float4 b4[kCh / 4];
    __shared__ int64_t pre[kMaxImages + 1];
    for (int i = threadIdx.x; i < kInW; i += blockDim.x) {
        int const k = i / kCh, co = i - k * kCh;
        reinterpret_cast<float*>(w4[k])[co] = params[kOffIn + co * kTaps * 2 + k];
    }
    for (int i = threadIdx.x; i < kCh; i += blockDim.x) reinterpret_cast<float*>(b4)[i] = params[kOffIn + kInW + i];
    after_previous(feat);
    // A thread forms eight channels (chunk c, four neighbouring lanes a pixel) of
    // kIncRun pixels in a row: their windows slide over one another, each weight
    // read from shared memory serves all of them, and a warp stores whole pixels.
    // Each channel's sum is bias, then the 18 inputs in order.
    scan_active(
        t.nimg,
        [&](int k) { return image_active(t, k) ? (t.px_base[k + 1] - t.px_base[k] + kIncRun - 1) / kIncRun : int64_t(0); },
        pre);
    walk_range(pre, t.nimg, kChunks, [&](int im, int e) {
        Img const o = t.img[im];
        int const P = o.w + 2;
        int const npx = P * (o.h + 2);
        int const g0 = e / kChunks * kIncRun, c = e % kChunks;
        bool inside[kIncRun];
        {
            int y = g0 / P, x = g0 - y * P;
#pragma unroll
            for (int u = 0; u < kIncRun; ++u) {
                inside[u] = !(y == 0 || x == 0 || y > o.h || x > o.w);
                if (++x == P) {
                    x = 0;
                    ++y;
                }
            }
        }
        float2 const* f2 = reinterpret_cast<float2 const*>(feat) + o.offset;
        // window columns g0-1 .. g0+kIncRun of the rows above, at and below
        float2 win[3][kIncRun + 2];
#pragma unroll
        for (int dy = 0; dy < 3; ++dy)
#pragma unroll
            for (int k = 0; k < kIncRun + 2; ++k) {
                int const g = g0 + (dy - 1) * P + (k - 1);
                win[dy][k] = g >= 0 && g < npx ? __ldg(f2 + g) : make_float2(0.0f, 0.0f);
            }
        Float2x a[kIncRun][4];
        float4 const b0 = b4[2 * c], b1 = b4[2 * c + 1];
#pragma unroll
        for (int u = 0; u < kIncRun; ++u) {
            a[u][0] = pair2(b0.x, b0.y);
            a[u][1] = pair2(b0.z, b0.w);
            a[u][2] = pair2(b1.x, b1.y);
            a[u][3] = pair2(b1.z, b1.w);
        }
#pragma unroll
        for (int k = 0; k < kTaps * 2; ++k) {
            float4 const w0 = w4[k][2 * c], w1 = w4[k][2 * c + 1];
            Float2x const w[4] = {pair2(w0.x, w0.y), pair2(w0.z, w0.w), pair2(w1.x, w1.y), pair2(w1.z, w1.w)};
#pragma unroll
            for (int u = 0; u < kIncRun; ++u) {
                float2 const in = win[(k / 2) / 3][(k / 2) % 3 + u];
                float const f = k % 2 == 0 ? in.x : in.y;
                Float2x const v = pair2(f, f);
#pragma unroll
                for (int i = 0; i < 4; ++i) a[u][i] = fma2(w[i], v, a[u][i]);
            }
        }
        uint4* dst = reinterpret_cast<uint4*>(out + (o.offset + g0) * kCh) + c;
#pragma unroll
        for (int u = 0; u < kIncRun; ++u) {
            if (g0 + u >= npx) continue;
            float r[8];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float2 const q = split2(a[u][i]);
                r[2 * i] = inside[u] ? fmaxf(q.x, 0.0f) : 0.0f;
                r[2 * i + 1] = inside[u] ? fmaxf(q.y, 0.0f) : 0.0f;
            }
            dst[u * kChunks] = pack8(r);
        }
    });
}

// Output convolution 32 -> 1 (+ bias), FP32 out, zero border.
__global__ void __launch_bounds__(256) out_forward_kernel(const __grid_constant__ Table t, bf16 const* in,
                                                          float const* params, float* out)
{
    after_previous(in);
    __shared__ float w[kOutW + 1];
    __shared__ int64_t pre[kMaxImages + 1];
    for (int i = threadIdx.x; i < kOutW + 1; i += blockDim.x) w[i] = params[kOffOut + i];
    walk_active(t, pre, 1, [&](int im, int g) {
        Img const o = t.img[im];
        int const P = o.w + 2;
        int const y = g / P, x = g - y * P;
        float a = 0.0f;
        if (!(y == 0 || x == 0 || y > o.h || x > o.w)) {
            a = w[kOutW];
            uint4 const* src = reinterpret_cast<uint4 const*>(in) + o.offset * kChunks;
#pragma unroll 3
            for (int tap = 0; tap < kTaps; ++tap) {
                int const q = g + (tap / 3 - 1) * P + (tap % 3 - 1);
                uint4 v[kChunks];
#pragma unroll
                for (int c = 0; c < kChunks; ++c) v[c] = __ldg(src + static_cast<int64_t>(q) * kChunks + c);
#pragma unroll
                for (int c = 0; c < kChunks; ++c) {
                    float f[8];
                    unpack8(v[c], f);
#pragma unroll
                    for (int e = 0; e < 8; ++e) a = __fmaf_rn(w[tap * kCh + c * 8 + e], f[e], a);
                }
            }
        }
        out[o.offset + g] = a;
    });
}

// Data gradient of the output convolution: dg[p][ci] = sum_tap du[p - tap] w[tap][ci].
__global__ void out_backward_data_kernel(const __grid_constant__ Table t, float const* du, float const* params, float* dg)
{
    after_previous(du);
    int const im = blockIdx.y;
    if (im >= t.nimg) return;
    Img const o = t.img[im];
    int64_t const P = o.w + 2, npx = P * (o.h + 2);
    int64_t const g = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (g >= npx) return;
    int64_t const y = g / P, x = g - y * P;
    float acc[kCh];
    for (int i = 0; i < kCh; ++i) acc[i] = 0.0f;
    if (!(y == 0 || x == 0 || y > o.h || x > o.w)) {
        float const* w = params + kOffOut;
        for (int tap = 0; tap < kTaps; ++tap) {
            float const d = du[o.offset + g - (tap / 3 - 1) * P - (tap % 3 - 1)];
            for (int ci = 0; ci < kCh; ++ci) acc[ci] = acc[ci] + d * w[tap * kCh + ci];
        }
    }
    float4* dst = reinterpret_cast<float4*>(dg + (o.offset + g) * kCh);
    for (int q = 0; q < 8; ++q) dst[q] = make_float4(acc[4 * q], acc[4 * q + 1], acc[4 * q + 2], acc[4 * q + 3]);
}

// Weight gradients of the thin convolutions (2 -> 32 input, 32 -> 1 output).
//
// Each is a sum over pixels of a 32-channel vector times a small window of
// the other tensor, so a warp holds the 32 channels in its lanes and every
// (tap, thin channel) weight of its lane in registers; it walks 16 consecutive
// pixels of a 128-pixel tile with the window sliding through registers, one
// coalesced channel load and nine (18) FMAs per pixel.  The tile's three
// window rows are staged in shared memory; a tile is a flat run of padded
// pixels, whose border pixels carry zero channels, so no pixel needs its
// coordinates.  Blocks keep their sums over all their tiles, add the eight
// warps' in order and write one partial each; reduce_parts_kernel adds those
// in order (deterministic).  Bound by the latency of the one pass over the
// channels: with a thread per weight walking 1,024 pixels in series the input
// and output gradients took 1,117 and 595 us of a 2,685 us gradient of eight
// 256^2 samples; here 14.8 and 10.7 us of 1,134.
constexpr int kThinBlock = 256;
constexpr int kThinWarps = kThinBlock / 32;
constexpr int kThinRun = kTilePx / kThinWarps;  // pixels per warp and tile

// Adds the block's per-lane sums over its warps; dst[v * 32 + lane].
template <int NV>
__device__ __forceinline__ void thin_block_sum(float const (&acc)[NV], float* smem, float (&sum)[(NV + 7) / 8])
{
    int const warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __syncthreads();
#pragma unroll
    for (int v = 0; v < NV; ++v) smem[(warp * NV + v) * 32 + lane] = acc[v];
    __syncthreads();
#pragma unroll
    for (int r = 0; r < (NV + 7) / 8; ++r) {
        int const v = warp + r * kThinWarps;
        float t = 0.0f;
        if (v < NV)
            for (int w = 0; w < kThinWarps; ++w) t = t + smem[(w * NV + v) * 32 + lane];
        sum[r] = t;
    }
}

// part[b][tap*32 + ci] = sum_q in[q][ci] du[q - tap], part[b][288] = sum_q du[q], over the block's tiles.
__global__ void __launch_bounds__(kThinBlock) out_wgrad_kernel(const __grid_constant__ Table t, float const* du,
                                                               bf16 const* in, float* part)
{
    constexpr int NV = kTaps + 1;
    __shared__ float win[3][kHalo + 2];
    __shared__ float red[kThinWarps * NV * 32];
    after_previous(du, in);
    int const warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float acc[NV] = {};
    for (int tile = blockIdx.x; tile < t.tile_base[t.nimg]; tile += gridDim.x) {
        int const im = find_image(t, tile);
        Img const o = t.img[im];
        int const P = o.w + 2, npx = P * (o.h + 2), end = P * (o.h + 1);
        int const start = P + (tile - t.tile_base[im]) * kTilePx;
        __syncthreads();
        for (int i = threadIdx.x; i < 3 * kHalo; i += kThinBlock) {
            int const r = i / kHalo, j = i - r * kHalo, g = start + (r - 1) * P - 1 + j;
            win[r][j] = g >= 0 && g < npx ? du[o.offset + g] : 0.0f;
        }
        __syncthreads();
        int const m0 = warp * kThinRun;
        bf16 const* src = in + (o.offset + start + m0) * kCh + lane;
        float d[3][3];
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            d[r][1] = win[r][m0];
            d[r][2] = win[r][m0 + 1];
        }
#pragma unroll
        for (int m = 0; m < kThinRun; ++m) {
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                d[r][0] = d[r][1];
                d[r][1] = d[r][2];
                d[r][2] = win[r][m0 + m + 2];
            }
            float const v = start + m0 + m < end ? __bfloat162float(src[m * kCh]) : 0.0f;
            // du at q - tap: the window read backwards
#pragma unroll
            for (int tap = 0; tap < kTaps; ++tap) acc[tap] = __fmaf_rn(v, d[2 - tap / 3][2 - tap % 3], acc[tap]);
            if (start + m0 + m < end) acc[kTaps] = acc[kTaps] + d[1][1];
        }
    }
    float sum[(NV + 7) / 8];
    thin_block_sum<NV>(acc, red, sum);
    float* dst = part + static_cast<int64_t>(blockIdx.x) * (kOutW + 1);
#pragma unroll
    for (int r = 0; r < (NV + 7) / 8; ++r) {
        int const v = warp + r * kThinWarps;
        if (v < kTaps) dst[v * kCh + lane] = sum[r];
        else if (v == kTaps && lane == 0) dst[kOutW] = sum[r];
    }
}

// part[b][(co*9 + tap)*2 + ci] = sum_p dz[p][co] feat[p + tap][ci], then the 32 bias sums, with
// dz = dh * (h > 0), over the block's tiles.
__global__ void __launch_bounds__(kThinBlock) inc_wgrad_kernel(const __grid_constant__ Table t, float const* dh,
                                                               bf16 const* h, float const* feat, float* part)
{
    constexpr int NV = 2 * kTaps + 1;
    __shared__ float2 win[3][kHalo + 2];
    __shared__ float red[kThinWarps * NV * 32];
    after_previous(dh, h, feat);
    int const warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float acc[NV] = {};
    for (int tile = blockIdx.x; tile < t.tile_base[t.nimg]; tile += gridDim.x) {
        int const im = find_image(t, tile);
        Img const o = t.img[im];
        int const P = o.w + 2, npx = P * (o.h + 2), end = P * (o.h + 1);
        int const start = P + (tile - t.tile_base[im]) * kTilePx;
        __syncthreads();
        for (int i = threadIdx.x; i < 3 * kHalo; i += kThinBlock) {
            int const r = i / kHalo, j = i - r * kHalo, g = start + (r - 1) * P - 1 + j;
            win[r][j] = g >= 0 && g < npx ? reinterpret_cast<float2 const*>(feat)[o.offset + g] : make_float2(0.0f, 0.0f);
        }
        __syncthreads();
        int const m0 = warp * kThinRun;
        int64_t const px = (o.offset + start + m0) * kCh + lane;
        // every load of the run in flight before the first use
        float dz[kThinRun];
        bf16 hv[kThinRun];
#pragma unroll
        for (int m = 0; m < kThinRun; ++m) {
            bool const in = start + m0 + m < end;
            dz[m] = in ? __ldg(dh + px + m * kCh) : 0.0f;
            hv[m] = in ? h[px + m * kCh] : __float2bfloat16_rn(0.0f);
        }
        float2 f[3][3];
#pragma unroll
        for (int r = 0; r < 3; ++r) {
            f[r][1] = win[r][m0];
            f[r][2] = win[r][m0 + 1];
        }
#pragma unroll
        for (int m = 0; m < kThinRun; ++m) {
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                f[r][0] = f[r][1];
                f[r][1] = f[r][2];
                f[r][2] = win[r][m0 + m + 2];
            }
            float const d = __bfloat162float(hv[m]) > 0.0f ? dz[m] : 0.0f;
#pragma unroll
            for (int tap = 0; tap < kTaps; ++tap) {
                acc[2 * tap] = __fmaf_rn(d, f[tap / 3][tap % 3].x, acc[2 * tap]);
                acc[2 * tap + 1] = __fmaf_rn(d, f[tap / 3][tap % 3].y, acc[2 * tap + 1]);
            }
            acc[2 * kTaps] = acc[2 * kTaps] + d;
        }
    }
    float sum[(NV + 7) / 8];
    thin_block_sum<NV>(acc, red, sum);
    float* dst = part + static_cast<int64_t>(blockIdx.x) * (kInW + kCh);
#pragma unroll
    for (int r = 0; r < (NV + 7) / 8; ++r) {
        int const v = warp + r * kThinWarps;
        if (v < 2 * kTaps) dst[lane * 2 * kTaps + v] = sum[r];
        else if (v == 2 * kTaps) dst[kInW + lane] = sum[r];
    }
}

// ------------------------------------------------------------------ level adjoints

// dfine[p] += 0.25 * dcoarse[parent(p)] (adjoint of the 2x2 average pool).
__global__ void pool_adjoint_kernel(const __grid_constant__ Table t, float const* dcoarse, float* dfine)
{
    after_previous(dcoarse);
    // t.img: fine level; t.aux: coarse level
    int const im = blockIdx.y;
    if (im >= t.nimg) return;
    Img const f = t.img[im], c = t.aux[im];
    int64_t const P = f.w + 2;
    int64_t const idx = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    int64_t const g = idx / 8;
    int const ch = static_cast<int>(idx % 8) * 4;
    if (g >= P * (f.h + 2)) return;
    int64_t const y = g / P, x = g - y * P;
    if (y == 0 || x == 0 || y > f.h || x > f.w) return;
    int64_t const cp = c.offset + ((y - 1) / 2 + 1) * (c.w + 2) + ((x - 1) / 2 + 1);
    float4 const d = *reinterpret_cast<float4 const*>(dcoarse + cp * kCh + ch);
    float4* o = reinterpret_cast<float4*>(dfine + (f.offset + g) * kCh + ch);
    float4 v = *o;
    v.x = v.x + 0.25f * d.x;
    v.y = v.y + 0.25f * d.y;
    v.z = v.z + 0.25f * d.z;
    v.w = v.w + 0.25f * d.w;
    *o = v;
}

// Adjoint of skip + up(coarse): dskip[p] += dx[p]; dcoarse[q] += sum of dx over q's children.
__global__ void upadd_adjoint_skip_kernel(const __grid_constant__ Table t, float const* dx, float* dskip)
{
    after_previous(dx);
    int const im = blockIdx.y;
    if (im >= t.nimg) return;
    Img const f = t.img[im];
    int64_t const P = f.w + 2;
    int64_t const idx = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    int64_t const g = idx / 8;
    int const ch = static_cast<int>(idx % 8) * 4;
    if (g >= P * (f.h + 2)) return;
    int64_t const q = (f.offset + g) * kCh + ch;
    float4 const d = *reinterpret_cast<float4 const*>(dx + q);
    float4* o = reinterpret_cast<float4*>(dskip + q);
    float4 v = *o;
    v.x = v.x + d.x;
    v.y = v.y + d.y;
    v.z = v.z + d.z;
    v.w = v.w + d.w;
    *o = v;
}

__global__ void upadd_adjoint_coarse_kernel(const __grid_constant__ Table t, float const* dx, float* dcoarse)
{
    after_previous(dx);
    // t.img: coarse level; t.aux: fine level
    int const im = blockIdx.y;
    if (im >= t.nimg) return;
    Img const c = t.img[im], f = t.aux[im];
    int64_t const P = c.w + 2;
    int64_t const idx = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    int64_t const g = idx / 8;
    int const ch = static_cast<int>(idx % 8) * 4;
    if (g >= P * (c.h + 2)) return;
    int64_t const y = g / P, x = g - y * P;
    if (y == 0 || x == 0 || y > c.h || x > c.w) return;
    int64_t const Pf = f.w + 2;
    float4 sacc = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int a = 0; a < 2; ++a)
        for (int b = 0; b < 2; ++b) {
            int64_t const fy = 2 * (y - 1) + a, fx = 2 * (x - 1) + b;  // interior coordinates
            if (fy >= f.h || fx >= f.w) continue;
            float4 const d = *reinterpret_cast<float4 const*>(dx + (f.offset + (fy + 1) * Pf + fx + 1) * kCh + ch);
            sacc.x = sacc.x + d.x;
            sacc.y = sacc.y + d.y;
            sacc.z = sacc.z + d.z;
            sacc.w = sacc.w + d.w;
        }
    float4* o = reinterpret_cast<float4*>(dcoarse + (c.offset + g) * kCh + ch);
    float4 v = *o;
    v.x = v.x + sacc.x;
    v.y = v.y + sacc.y;
    v.z = v.z + sacc.z;
    v.w = v.w + sacc.w;
    *o = v;
}

// dst = src over every pixel of the table's images (16 bytes per thread).
__global__ void copy_act_kernel(const __grid_constant__ Table t, bf16 const* src, bf16* dst)
{
    __shared__ int64_t pre[kMaxImages + 1];
    walk_active(t, pre, kChunks, [&](int im, int idx) {
        int64_t const q = t.img[im].offset * kChunks + idx;
        reinterpret_cast<uint4*>(dst)[q] = reinterpret_cast<uint4 const*>(src)[q];
    });
}

// Decoder input of the inference pass: skip + nearest-upsampled coarse
// features summed in FP32 and stored in BF16 (zero border), so the decoder
// convolution reads one operand through the pipelined plain mode.  (The
// training pass keeps the two operands, which the tensor core sums in FP32,
// because the weight gradient needs them apart.)
// A thread per 16-byte chunk, as pool_kernel (33 -> 31 us at 1 M pixels,
// 10.5 -> 5.2 at 64 k).
__global__ void upadd_kernel(const __grid_constant__ Table t, bf16 const* skip, bf16 const* coarse, bf16* out)
{
    __shared__ int64_t pre[kMaxImages + 1];
    after_previous(skip, coarse);
    walk_active(t, pre, kChunks, [&](int im, int q) {
        Img const o = t.img[im], ci = t.aux[im];
        int const g = q / kChunks, c = q % kChunks, P = o.w + 2;
        int const y = g / P, x = g - y * P;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (!(y == 0 || x == 0 || y > o.h || x > o.w)) {
            int64_t const cpx = ci.offset + static_cast<int64_t>((y - 1) / 2 + 1) * (ci.w + 2) + ((x - 1) / 2 + 1);
            float f[8], a[8];
            unpack8(__ldg(reinterpret_cast<uint4 const*>(skip) + o.offset * kChunks + q), f);
            unpack8(__ldg(reinterpret_cast<uint4 const*>(coarse) + cpx * kChunks + c), a);
#pragma unroll
            for (int i = 0; i < 8; ++i) f[i] = f[i] + a[i];
            v = pack8(f);
        }
        reinterpret_cast<uint4*>(out)[o.offset * kChunks + q] = v;
    });
}

// ------------------------------------------------------------------ node-level wrapper (FP32)

struct Samples
{
    int n;
    Sample s[kMaxImages];
    Img top[kMaxImages];                 // level-0 network image of each sample
    int32_t item_base[kMaxImages + 1];   // first fused-wrapper work item of each sample
    int32_t strip_base[kMaxImages + 1];  // first CTA of strips of each sample
    int32_t strip_rows;                  // rows of a strip
    int const* active;                   // per sample: 0 = skip (NULL: all run)
};

__device__ __forceinline__ bool sample_active(Samples const& ss, int i)
{
    return ss.active == nullptr || __ldg(ss.active + i) != 0;
}

__device__ __forceinline__ bool node_of(Samples const& ss, int64_t& row, Sample& sm)
{
    sm = ss.s[blockIdx.y];
    row = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    return row < static_cast<int64_t>(sm.nx) * sm.ny;
}

// y = alpha * x + beta * dinv (b - K e)   with optional K e: general Jacobi-type update
// out = base + w * dinv * (b - K e)
__global__ void jacobi_kernel(const __grid_constant__ Samples ss, float const* nu, float const* dinv, float const* b,
                              float const* e, float const* base, float w, float* out)
{
    int64_t row;
    Sample sm;
    if (!node_of(ss, row, sm)) return;
    int64_t const o = sm.offset;
    float const ke = e != nullptr ? mag_apply_node(e + o, nu + o, sm.nx, sm.ny, row) : 0.0f;
    float const r = b[o + row] - ke;
    float const bv = base != nullptr ? base[o + row] : 0.0f;
    out[o + row] = bv + w * (dinv[o + row] * r);
}

// out = K e
__global__ void kapply_kernel(const __grid_constant__ Samples ss, float const* nu, float const* e, float* out)
{
    int64_t row;
    Sample sm;
    if (!node_of(ss, row, sm)) return;
    int64_t const o = sm.offset;
    out[o + row] = mag_apply_node(e + o, nu + o, sm.nx, sm.ny, row);
}

constexpr int kDotBlock = 256;

// Per-sample partial sums of up to three products a1.b1, a2.b2, a3.b3 (FP64).
__global__ void dots_kernel(const __grid_constant__ Samples ss, float const* a1, float const* b1, float const* a2,
                            float const* b2, float const* a3, float const* b3, double* part, int nblocks_x)
{
    __shared__ double red[3][kDotBlock / 32];
    Sample const sm = ss.s[blockIdx.y];
    int64_t const n = static_cast<int64_t>(sm.nx) * sm.ny;
    double acc[3] = {0.0, 0.0, 0.0};
    for (int64_t row = static_cast<int64_t>(blockIdx.x) * kDotBlock + threadIdx.x; row < n;
         row += static_cast<int64_t>(nblocks_x) * kDotBlock) {
        int64_t const q = sm.offset + row;
        acc[0] += static_cast<double>(a1[q]) * static_cast<double>(b1[q]);
        if (a2 != nullptr) acc[1] += static_cast<double>(a2[q]) * static_cast<double>(b2[q]);
        if (a3 != nullptr) acc[2] += static_cast<double>(a3[q]) * static_cast<double>(b3[q]);
    }
    for (int k = 0; k < 3; ++k) {
        double v = acc[k];
        for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
        if ((threadIdx.x & 31) == 0) red[k][threadIdx.x >> 5] = v;
    }
    __syncthreads();
    if (threadIdx.x < 3) {
        double v = 0.0;
        for (int w = 0; w < kDotBlock / 32; ++w) v += red[threadIdx.x][w];
        part[(static_cast<int64_t>(blockIdx.y) * nblocks_x + blockIdx.x) * 3 + threadIdx.x] = v;
    }
}

// dots[s][k] = sum over blocks (fixed order).
__global__ void dots_finish_kernel(double const* part, int nsamples, int nblocks_x, double* dots)
{
    int const i = threadIdx.x;
    if (i >= nsamples * 3) return;
    int const s = i / 3, k = i % 3;
    double v = 0.0;
    for (int b = 0; b < nblocks_x; ++b) v += part[(static_cast<int64_t>(s) * nblocks_x + b) * 3 + k];
    dots[i] = v;
}

// Feature image of the network's top level: 2x2 average of
// [D^-1/2 r1 / s, log(nu)/log(1000)] over the nodes of each half-resolution
// pixel (nodes outside the grid count as zero), s = rms(D^-1/2 r1).
__global__ void features_kernel(const __grid_constant__ Samples ss, const __grid_constant__ Table t, float const* r1,
                                float const* nu, float const* dinv, double const* dots, float const* lognu, float* feat)
{
    __shared__ int64_t pre[kMaxImages + 1];
    __shared__ float inv_rms[kMaxImages];   // 1 / rms(D^-1/2 r1) per sample
    after_previous(dots, r1);
    for (int k = threadIdx.x; k < ss.n; k += blockDim.x) {
        double const ms = dots[k * 3] / (static_cast<double>(ss.s[k].nx) * ss.s[k].ny);
        inv_rms[k] = ms > 0.0 ? static_cast<float>(1.0 / sqrt(ms)) : 0.0f;
    }
    float const inv_l = static_cast<float>(1.0 / log(1000.0));
    walk_active(t, pre, 1, [&](int im, int g) {
        int const sidx = t.sample[im];
        Sample const sm = ss.s[sidx];
        Img const o = t.img[im];
        int const P = o.w + 2;
        int const y = g / P, x = g - y * P;
        float f0 = 0.0f, f1 = 0.0f;
        if (!(y == 0 || x == 0 || y > o.h || x > o.w)) {
            float const inv_s = inv_rms[sidx];
            for (int a = 0; a < 2; ++a)
                for (int b = 0; b < 2; ++b) {
                    int64_t const j = 2 * (y - 1) + a, i = 2 * (x - 1) + b;
                    if (j >= sm.ny || i >= sm.nx) continue;
                    int64_t const q = sm.offset + j * sm.nx + i;
                    f0 = f0 + r1[q] * sqrtf(dinv[q]) * inv_s;
                    if (lognu == nullptr) f1 = f1 + logf(nu[q]) * inv_l;
                }
            f0 = f0 * 0.25f;
            f1 = lognu != nullptr ? lognu[o.offset + g] : f1 * 0.25f;
        }
        feat[2 * (o.offset + g)] = f0;
        feat[2 * (o.offset + g) + 1] = f1;
    });
}

// Gradient of the loss with respect to u:
// g = -(2 ub uKu b - 2 ub^2 Ku) / (uKu^2 xb) / nsamples.
__global__ void loss_grad_u_kernel(const __grid_constant__ Samples ss, float const* b, float const* ku,
                                   double const* dots_u, double const* dots_x, float* gu)
{
    int64_t row;
    Sample sm;
    if (!node_of(ss, row, sm)) return;
    double const ub = dots_u[blockIdx.y * 3], uku = dots_u[blockIdx.y * 3 + 1], xb = dots_x[blockIdx.y * 3];
    double const den = uku * uku * xb * ss.n;
    double const cb = den > 0 ? -2.0 * ub * uku / den : 0.0;
    double const ck = den > 0 ? 2.0 * ub * ub / den : 0.0;
    int64_t const q = sm.offset + row;
    gu[q] = static_cast<float>(cb * b[q] + ck * ku[q]);
}

// g_net[top pixel] = s * sum over interior child nodes of D^-1/2 g_e2.
__global__ void net_grad_kernel(const __grid_constant__ Samples ss, float const* ge2, float const* dinv,
                                double const* dots, float* gnet)
{
    int const sidx = blockIdx.y;
    Sample const sm = ss.s[sidx];
    Img const o = ss.top[sidx];
    int64_t const P = o.w + 2, npx = P * (o.h + 2);
    int64_t const g = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (g >= npx) return;
    int64_t const y = g / P, x = g - y * P;
    float v = 0.0f;
    if (!(y == 0 || x == 0 || y > o.h || x > o.w)) {
        double const ms = dots[sidx * 3] / (static_cast<double>(sm.nx) * sm.ny);
        float const s = static_cast<float>(sqrt(ms));
        float acc = 0.0f;
        for (int a = 0; a < 2; ++a)
            for (int b = 0; b < 2; ++b) {
                int64_t const j = 2 * (y - 1) + a, i = 2 * (x - 1) + b;
                if (j >= sm.ny || i >= sm.nx) continue;
                if (i == 0 || j == 0 || i + 1 == sm.nx || j + 1 == sm.ny) continue;
                int64_t const q = sm.offset + j * sm.nx + i;
                acc = acc + sqrtf(dinv[q]) * ge2[q];
            }
        v = s * acc;
    }
    gnet[o.offset + g] = v;
}

// out = a x + b y
__global__ void axpby_kernel(const __grid_constant__ Samples ss, float a, float const* x, float b, float const* y,
                             float* out)
{
    int64_t row;
    Sample sm;
    if (!node_of(ss, row, sm)) return;
    int64_t const q = sm.offset + row;
    out[q] = a * x[q] + b * y[q];
}

// ------------------------------------------------------------------ fused wrapper passes
//
// Work items of kWrapRows consecutive nodes of one sample, so no block idles
// on the small grids of a batch of uneven sizes; 32-bit index arithmetic.

constexpr int kWrapRows = 2048;

struct WrapItem
{
    int32_t sample, begin, end, index;   // index: item number within its sample
};

__device__ __forceinline__ double block_sum_d(double v, double* red)
{
    for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    double t = 0.0;
    if (threadIdx.x == 0)
        for (int w = 0; w < static_cast<int>(blockDim.x) / 32; ++w) t += red[w];
    return t;
}

// Prefix of the active samples' wrapper items (the items of a sample are
// contiguous from item_base) and the item of active unit a.
__device__ __forceinline__ int scan_items(Samples const& ss, int64_t* pre)
{
    scan_active(
        ss.n, [&](int k) { return sample_active(ss, k) ? int64_t(ss.item_base[k + 1] - ss.item_base[k]) : int64_t(0); },
        pre);
    return static_cast<int>(pre[ss.n]);
}

__device__ __forceinline__ int item_of(Samples const& ss, int64_t const* pre, int a)
{
    int const k = find_unit(pre, ss.n, a);
    return ss.item_base[k] + (a - static_cast<int>(pre[k]));
}

// The active samples' CTAs of strips (mag_ops.cuh): f(sample, strip, j0, j1, c0,
// cta) for the calling warp's strip of every CTA it is handed; `after(cta)` runs
// for the whole block after each.
template <class F, class A>
__device__ __forceinline__ void walk_strips(Samples const& ss, int64_t* pre, F const& f, A const& after)
{
    scan_active(
        ss.n, [&](int k) { return sample_active(ss, k) ? int64_t(ss.strip_base[k + 1] - ss.strip_base[k]) : int64_t(0); },
        pre);
    int const nact = static_cast<int>(pre[ss.n]);
    for (int a = blockIdx.x; a < nact; a += gridDim.x) {
        int const k = find_unit(pre, ss.n, a), within = a - static_cast<int>(pre[k]);
        Sample const sm = ss.s[k];
        Strips const st = strips_of(sm.nx, sm.ny, ss.strip_rows);
        int const strip = within * kStripWarps + static_cast<int>(threadIdx.x >> 5);
        if (strip < st.count) {
            int const block = strip / st.strips, j0 = block * st.rows;
            f(sm, (strip - block * st.strips) * kStripCols, j0, min(sm.ny, j0 + st.rows));
        }
        after(ss.strip_base[k] + within);
    }
}

// Operand e1 = w D^-1 r.
struct WrapPreSrc
{
    struct Raw
    {
        float d, r;
    };
    struct Own
    {};
    float const* __restrict__ d;
    float const* __restrict__ r;
    __device__ __forceinline__ Raw load(int row) const { return {d[row], r[row]}; }
    __device__ __forceinline__ Own own(int) const { return {}; }
    __device__ __forceinline__ float value(Raw const& v) const { return kOmega * (v.d * v.r); }
};

// r1 = r - K e1 with e1 = w D^-1 r formed on the fly (boundary rows: r1 = r - e1),
// and the partial sums of |D^-1/2 r1|^2 per CTA of strips.  B200, 4.1 M nodes: a
// thread per node with its own stencil 31 us, strips 17.
__global__ void __launch_bounds__(256) wrap_pre_kernel(const __grid_constant__ Samples ss, float const* nu,
                                                       float const* dinv, float const* r, float* r1, double* part)
{
    __shared__ double red[8];
    __shared__ int64_t pre[kMaxImages + 1];
    double acc = 0.0;
    after_previous(r);
    walk_strips(
        ss, pre,
        [&](Sample const& sm, int c0, int j0, int j1) {
            float* out = r1 + sm.offset;
            mag2d_strip<float>(WrapPreSrc {dinv + sm.offset, r + sm.offset}, nu + sm.offset, sm.nx, sm.ny, c0, j0, j1,
                               [&](int row, float q, float, WrapPreSrc::Raw const& raw, WrapPreSrc::Own) {
                                   float const v = raw.r - q;
                                   out[row] = v;
                                   acc += static_cast<double>(raw.d) * static_cast<double>(v) * static_cast<double>(v);
                               });
        },
        [&](int cta) {
            double const t = block_sum_d(acc, red);
            if (threadIdx.x == 0) part[cta] = t;
            acc = 0.0;
        });
}

// dots[s*3] = sum of the sample's item partials: one warp per sample, each
// lane summing a fixed strided subset in order, then a fixed butterfly
// (deterministic for a given batch geometry).
__global__ void wrap_finish_kernel(const __grid_constant__ Samples ss, double const* part, double* dots)
{
    int const sidx = blockIdx.x;
    after_previous(part);
    if (sidx >= ss.n || !sample_active(ss, sidx)) return;
    double t = 0.0;
    for (int k = ss.strip_base[sidx] + static_cast<int>(threadIdx.x); k < ss.strip_base[sidx + 1]; k += 32) t += part[k];
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (threadIdx.x == 0) dots[sidx * 3] = t;
}

// s = rms(D^-1/2 r1) per sample (dots[k*3] = |D^-1/2 r1|^2), staged in shared
// memory before a walk (whose scan barrier publishes it).
__device__ __forceinline__ void stage_rms(Samples const& ss, double const* dots, float* sc)
{
    for (int k = threadIdx.x; k < ss.n; k += blockDim.x)
        sc[k] = static_cast<float>(sqrt(dots[k * 3] / (static_cast<double>(ss.s[k].nx) * ss.s[k].ny)));
}

// dinv = 1 / diag(K) (identity on the boundary); nu given per node.
__global__ void __launch_bounds__(256) dinv_kernel(const __grid_constant__ Samples ss, WrapItem const* items,
                                                   float const* __restrict__ nu, float* __restrict__ dinv)
{
    WrapItem const it = items[blockIdx.x];
    Sample const sm = ss.s[it.sample];
    int const nx = sm.nx, ny = sm.ny;
    float const* v = nu + sm.offset;
    float* o = dinv + sm.offset;
#pragma unroll 4
    for (int row = it.begin + static_cast<int>(threadIdx.x); row < it.end; row += 256) {
        int const j = row / nx, i = row - j * nx;
        bool const in = !(i == 0 || j == 0 || i + 1 == nx || j + 1 == ny);
        float const below = v[j >= 2 ? row - nx : row], left = v[i >= 2 ? row - 1 : row], c = v[row];
        float d = 0.0f;
        if (j >= 2) d = d + below;
        d = d + c;
        if (i >= 2) d = d + left;
        d = d + c;
        o[row] = in ? 1.0f / d : 1.0f;
    }
}

// e2 = w D^-1 r + s D^-1/2 up(unet) at interior nodes (w D^-1 r on the
// boundary), s = rms of the sample's D^-1/2 r1.  Items as wrap_pre.
__global__ void __launch_bounds__(256) wrap_e2_kernel(const __grid_constant__ Samples ss, WrapItem const* items,
                                                      float const* dinv, float const* r, float const* unet,
                                                      double const* dots, float* e2)
{
    __shared__ int64_t pre[kMaxImages + 1];
    __shared__ float sc[kMaxImages];
    after_previous(unet, dots);
    stage_rms(ss, dots, sc);
    int const nact = scan_items(ss, pre);
    for (int a = blockIdx.x; a < nact; a += gridDim.x) {
        WrapItem const it = items[item_of(ss, pre, a)];
        int const k = it.sample;
        Sample const sm = ss.s[k];
        int const nx = sm.nx, ny = sm.ny;
        float const* d_s = dinv + sm.offset;
        float const* r_s = r + sm.offset;
        Img const o = ss.top[k];
        float const* un = unet + o.offset;
        int const P = o.w + 2;
        float const s_k = sc[k];
        int row = it.begin + static_cast<int>(threadIdx.x);
        int j = row / nx, i = row - j * nx;
        for (; row < it.end; row += blockDim.x) {
            float v = kOmega * (d_s[row] * r_s[row]);
            if (!(i == 0 || j == 0 || i + 1 == nx || j + 1 == ny))
                v = v + s_k * sqrtf(d_s[row]) * un[(j / 2 + 1) * P + (i / 2 + 1)];
            e2[sm.offset + row] = v;
            i += blockDim.x;
            while (i >= nx) {
                i -= nx;
                ++j;
            }
        }
    }
}

// Operand e2, with D^-1 and r on the side.
struct WrapPostSrc
{
    using Raw = float;
    struct Own
    {
        float d, r;
    };
    float const* __restrict__ e;
    float const* __restrict__ d;
    float const* __restrict__ r;
    __device__ __forceinline__ Raw load(int row) const { return e[row]; }
    __device__ __forceinline__ Own own(int row) const { return {d[row], r[row]}; }
    __device__ __forceinline__ float value(Raw v) const { return v; }
};

// M(r) = e2 + w D^-1 (r - K e2) (boundary rows: K e2 -> e2), in strips as wrap_pre
// (24 -> 17.5 us).
__global__ void __launch_bounds__(256) wrap_post_kernel(const __grid_constant__ Samples ss, float const* nu,
                                                        float const* dinv, float const* r, float const* e2, float* out)
{
    __shared__ int64_t pre[kMaxImages + 1];
    after_previous(e2);
    walk_strips(
        ss, pre,
        [&](Sample const& sm, int c0, int j0, int j1) {
            float* o = out + sm.offset;
            mag2d_strip<float>(WrapPostSrc {e2 + sm.offset, dinv + sm.offset, r + sm.offset}, nu + sm.offset, sm.nx, sm.ny,
                               c0, j0, j1, [&](int row, float q, float e0, float, WrapPostSrc::Own const& w) {
                                   o[row] = e0 + kOmega * (w.d * (w.r - q));
                               });
        },
        [](int) {});
}

// log(nu) / log(1000), pooled 2 x 2 onto the top-level image of every sample
// (the network's second input channel; zero on the image border).
__global__ void lognu_feature_kernel(const __grid_constant__ Samples ss, const __grid_constant__ Table t, float const* nu,
                                     float* lognu)
{
    __shared__ int64_t pre[kMaxImages + 1];
    float const inv_l = static_cast<float>(1.0 / log(1000.0));
    walk_active(t, pre, 1, [&](int im, int g) {
        Sample const sm = ss.s[t.sample[im]];
        Img const o = t.img[im];
        int const P = o.w + 2;
        int const y = g / P, x = g - y * P;
        float f1 = 0.0f;
        if (!(y == 0 || x == 0 || y > o.h || x > o.w)) {
            for (int a = 0; a < 2; ++a)
                for (int b = 0; b < 2; ++b) {
                    int64_t const j = 2 * (y - 1) + a, i = 2 * (x - 1) + b;
                    if (j >= sm.ny || i >= sm.nx) continue;
                    f1 = f1 + logf(nu[sm.offset + j * sm.nx + i]) * inv_l;
                }
            f1 = f1 * 0.25f;
        }
        lognu[o.offset + g] = f1;
    });
}

__global__ void adam_kernel(float* p, float const* g, float* m, float* v, int n, float lr, float b1t, float b2t)
{
    int const i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float const gi = g[i];
    float const mi = 0.9f * m[i] + 0.1f * gi;
    float const vi = 0.999f * v[i] + 0.001f * gi * gi;
    m[i] = mi;
    v[i] = vi;
    float const mh = mi / b1t, vh = vi / b2t;
    p[i] = p[i] - lr * mh / (sqrtf(vh) + 1e-8f);
}

// ------------------------------------------------------------------ host side

struct DevBuf
{
    void* p = nullptr;
    size_t bytes = 0;
    ~DevBuf() { cudaFree(p); }
    sil_status alloc(size_t b)
    {
        if (b <= bytes) return SIL_OK;
        cudaFree(p);
        p = nullptr;
        bytes = 0;
        cudaError_t const e = cudaMalloc(&p, std::max<size_t>(b, 256));
        if (e != cudaSuccess) return cuda_fail(e, "precond workspace");
        bytes = b;
        return SIL_OK;
    }
    template <class T>
    T* as() const { return static_cast<T*>(p); }
};

// Geometry of one network level for the images that reach it.
struct Level
{
    std::vector<int> images;       // sample indices present
    std::vector<Img> img;          // per present image (same order)
    int64_t npx = 0;               // padded pixels of the level buffer
    int ntiles = 0;
};

class Workspace
{
public:
    std::vector<Sample> samples;
    int64_t nodes = 0;
    std::vector<Level> levels;
    std::vector<int> depth;        // levels per sample
    Samples ss {};
    // node-level FP32 vectors
    DevBuf dinv, r1, e2, u, ku, tmp, gu, ge2;
    DevBuf lognu;                  // top-level log(nu) feature channel of a fixed nu (set_static_nu)
    float const* lognu_for = nullptr;  // the nu it was formed from (NULL: none)
    DevBuf dparts;                 // per-sample dot partials
    DevBuf dots;                   // [3 sets][nsamples][3]
    int dot_blocks = 0;
    // network buffers per level
    std::vector<DevBuf> h, p, g, pin, dh, dg, dx;
    DevBuf taps;                   // 9 x level-0 pixels: output-convolution partials
    DevBuf feat, unet, gnet;
    DevBuf witems, wpart;          // fused wrapper work items and their partial sums
    int nwitems = 0;
    int nstrips = 0;               // CTAs of strips
    DevBuf wparts;                 // weight-gradient partials
    int wgrad_grid = 0;
    int thin_grid = 0;
    int64_t max_node_per_sample = 0;
    int const* active = nullptr;   // per-sample switch of the current forward (NULL: all)

    sil_status build(std::vector<Sample> const& s);
    Table table(int level, int aux_level, bool aux_is_finer) const;
};

static int depth_of(int h, int w)
{
    int d = 1;
    while (std::min(h, w) >= 16) {
        h = (h + 1) / 2;
        w = (w + 1) / 2;
        ++d;
    }
    return d;
}

sil_status Workspace::build(std::vector<Sample> const& s)
{
    samples = s;
    int const n = static_cast<int>(s.size());
    if (n < 1 || n > kMaxImages) return fail(SIL_ERR_INVALID, "precond: 1 to 64 samples per batch");
    nodes = 0;
    max_node_per_sample = 0;
    depth.assign(n, 0);
    int maxd = 0;
    ss = Samples {};
    ss.n = n;
    for (int i = 0; i < n; ++i) {
        if (s[i].nx < 3 || s[i].ny < 3) return fail(SIL_ERR_INVALID, "precond: grids need at least 3x3 nodes");
        if (static_cast<int64_t>(s[i].nx) * s[i].ny >= (int64_t(1) << 31))
            return fail(SIL_ERR_INVALID, "precond: a grid must have fewer than 2^31 nodes");
        ss.s[i] = s[i];
        nodes = std::max<int64_t>(nodes, s[i].offset + static_cast<int64_t>(s[i].nx) * s[i].ny);
        max_node_per_sample = std::max<int64_t>(max_node_per_sample, static_cast<int64_t>(s[i].nx) * s[i].ny);
        depth[i] = depth_of((s[i].ny + 1) / 2, (s[i].nx + 1) / 2);
        maxd = std::max(maxd, depth[i]);
    }
    levels.assign(maxd, Level {});
    for (int l = 0; l < maxd; ++l) {
        Level& L = levels[l];
        for (int i = 0; i < n; ++i) {
            if (depth[i] <= l) continue;
            int hh = (s[i].ny + 1) / 2, ww = (s[i].nx + 1) / 2;
            for (int k = 0; k < l; ++k) {
                hh = (hh + 1) / 2;
                ww = (ww + 1) / 2;
            }
            L.images.push_back(i);
            L.img.push_back({hh, ww, L.npx});
            L.npx += static_cast<int64_t>(hh + 2) * (ww + 2);
            L.ntiles += static_cast<int>((static_cast<int64_t>(ww + 2) * hh + kTilePx - 1) / kTilePx);
        }
    }
    for (int i = 0; i < n; ++i) ss.top[i] = levels[0].img[i];
    size_t const nb = static_cast<size_t>(nodes) * sizeof(float);
    for (DevBuf* b : {&dinv, &r1, &e2, &u, &ku, &tmp, &gu, &ge2}) {
        sil_status const st = b->alloc(nb);
        if (st != SIL_OK) return st;
    }
    dot_blocks = static_cast<int>(std::min<int64_t>(64, (max_node_per_sample + kDotBlock - 1) / kDotBlock));
    if (sil_status st = dparts.alloc(sizeof(double) * 3 * n * dot_blocks); st != SIL_OK) return st;
    if (sil_status st = dots.alloc(sizeof(double) * 3 * 3 * n); st != SIL_OK) return st;
    h.resize(maxd);
    pin.resize(maxd);
    p.resize(maxd);
    g.resize(maxd);
    dh.resize(maxd);
    dg.resize(maxd);
    dx.resize(maxd);
    // Every level buffer starts zeroed: no kernel writes the top and bottom
    // border rows of an image, which must read as zero.
    for (int l = 0; l < maxd; ++l) {
        size_t const a = static_cast<size_t>(levels[l].npx) * kCh;
        for (DevBuf* b : {&h[l], &p[l], &g[l], &pin[l]}) {
            if (sil_status st = b->alloc(a * sizeof(bf16)); st != SIL_OK) return st;
            SIL_CUDA_CHECK(cudaMemset(b->p, 0, a * sizeof(bf16)));
        }
        for (DevBuf* b : {&dh[l], &dg[l], &dx[l]}) {
            if (sil_status st = b->alloc(a * sizeof(float)); st != SIL_OK) return st;
            SIL_CUDA_CHECK(cudaMemset(b->p, 0, a * sizeof(float)));
        }
    }
    {
        std::vector<WrapItem> wi;
        for (int i = 0; i < n; ++i) {
            int const rows = s[i].nx * s[i].ny;
            int idx = 0;
            ss.item_base[i] = static_cast<int32_t>(wi.size());
            for (int b = 0; b < rows; b += kWrapRows, ++idx) wi.push_back({i, b, std::min(rows, b + kWrapRows), idx});
        }
        ss.item_base[n] = static_cast<int32_t>(wi.size());
        nwitems = static_cast<int>(wi.size());
        if (sil_status st = witems.alloc(sizeof(WrapItem) * wi.size()); st != SIL_OK) return st;
        // strips: one wave of two CTAs per multiprocessor before they get longer
        int dev = 0, sms = 148;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        for (ss.strip_rows = kStripBatch;; ss.strip_rows += kStripBatch) {
            nstrips = 0;
            for (int i = 0; i < n; ++i) {
                ss.strip_base[i] = nstrips;
                nstrips += strips_of(s[i].nx, s[i].ny, ss.strip_rows).ctas;
            }
            ss.strip_base[n] = nstrips;
            if (nstrips <= 2 * sms || ss.strip_rows >= 32) break;
        }
        if (sil_status st = wpart.alloc(sizeof(double) * nstrips); st != SIL_OK) return st;
        SIL_CUDA_CHECK(cudaMemcpy(witems.p, wi.data(), sizeof(WrapItem) * wi.size(), cudaMemcpyHostToDevice));
    }
    int64_t const top = levels[0].npx;
    if (sil_status st = taps.alloc(top * kTaps * sizeof(float)); st != SIL_OK) return st;
    SIL_CUDA_CHECK(cudaMemset(taps.p, 0, top * kTaps * sizeof(float)));
    if (sil_status st = feat.alloc(top * 2 * sizeof(float)); st != SIL_OK) return st;
    if (sil_status st = unet.alloc(top * sizeof(float)); st != SIL_OK) return st;
    if (sil_status st = gnet.alloc(top * sizeof(float)); st != SIL_OK) return st;
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    wgrad_grid = 2 * sms;
    thin_grid = 4 * sms;
    size_t const wp = std::max<size_t>(static_cast<size_t>(wgrad_grid) * kWgradParts,
                                       static_cast<size_t>(thin_grid) * (kInW + kCh));
    if (sil_status st = wparts.alloc(wp * sizeof(float)); st != SIL_OK) return st;
    return SIL_OK;
}

// Table of `level`; aux entries describe the same images at aux_level.
Table Workspace::table(int level, int aux_level, bool) const
{
    Table t {};
    Level const& L = levels[level];
    t.nimg = static_cast<int>(L.images.size());
    t.tile_base[0] = 0;
    t.active = active;
    t.px_base[0] = 0;
    for (int k = 0; k < t.nimg; ++k) {
        t.img[k] = L.img[k];
        t.sample[k] = L.images[k];
        t.px_base[k + 1] = t.px_base[k] + static_cast<int64_t>(L.img[k].h + 2) * (L.img[k].w + 2);
        int64_t const tiles = (static_cast<int64_t>(L.img[k].w + 2) * L.img[k].h + kTilePx - 1) / kTilePx;
        t.tile_base[k + 1] = t.tile_base[k] + static_cast<int32_t>(tiles);
        // (a batch of one-level images has no other level: aux stays empty)
        if (aux_level >= 0 && aux_level < static_cast<int>(levels.size())) {
            Level const& A = levels[aux_level];
            int const sidx = L.images[k];
            auto it = std::find(A.images.begin(), A.images.end(), sidx);
            t.aux[k] = it != A.images.end() ? A.img[it - A.images.begin()] : Img {0, 0, 0};
        }
    }
    return t;
}

namespace {

size_t conv_smem(int mode = kUpAdd)
{
    // kPlain and kUpAdd use both halo buffers (ring stages / two operands)
    return sizeof(ConvSmem) - (mode == kUpAdd || mode == kPlain ? 0 : sizeof(uint4) * kChunks * 3 * kHalo);
}
size_t wgrad_smem() { return sizeof(WgradSmem) + 1024; }

bool g_attr_done = false;
int g_sms = 0;  // multiprocessor count, read once (outside any stream capture)
int g_conv_per_sm[kModes] = {};  // resident conv CTAs per SM, by input mode
// Grid-stride kernels of the forward pass and their resident blocks per SM.
enum WalkKind { kWalkInc = 0, kWalkOut, kWalkGather, kWalkPool, kWalkCopy, kWalkFeat, kWalkPre, kWalkPost, kWalkLogNu,
                kWalkE2, kWalkUpAdd, kWalkKinds };
int g_walk_per_sm[kWalkKinds] = {1, 1, 1, 1, 1, 1, 1, 1, 1, 1, 1};

sil_status ensure_attributes()
{
    if (g_attr_done) return SIL_OK;
    int dev = 0;
    SIL_CUDA_CHECK(cudaGetDevice(&dev));
    SIL_CUDA_CHECK(cudaDeviceGetAttribute(&g_sms, cudaDevAttrMultiProcessorCount, dev));
    for (void const* k : {reinterpret_cast<void const*>(conv3x3_kernel), reinterpret_cast<void const*>(conv3x3_plain_kernel)}) {
        SIL_CUDA_CHECK(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(conv_smem())));
    }
    // all of the unified L1 / shared storage as shared memory, so several
    // CTAs of these shared-memory-heavy kernels fit on one multiprocessor
    SIL_CUDA_CHECK(cudaFuncSetAttribute(conv3x3_kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                        cudaSharedmemCarveoutMaxShared));
    SIL_CUDA_CHECK(cudaFuncSetAttribute(conv3x3_plain_kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                        cudaSharedmemCarveoutMaxShared));
    SIL_CUDA_CHECK(cudaFuncSetAttribute(wgrad_kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                        cudaSharedmemCarveoutMaxShared));
    // resident CTAs per multiprocessor from the kernel's registers and each
    // mode's shared memory (1 KB per CTA reserved by the runtime)
    cudaFuncAttributes fa {};
    cudaFuncAttributes fp {};
    SIL_CUDA_CHECK(cudaFuncGetAttributes(&fa, conv3x3_kernel));
    SIL_CUDA_CHECK(cudaFuncGetAttributes(&fp, conv3x3_plain_kernel));
    int smem_sm = 0, regs_sm = 0;
    SIL_CUDA_CHECK(cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev));
    SIL_CUDA_CHECK(cudaDeviceGetAttribute(&regs_sm, cudaDevAttrMaxRegistersPerMultiprocessor, dev));
    for (int m = 0; m < kModes; ++m) {
        int const by_smem = smem_sm / static_cast<int>(conv_smem(m) + 1024);
        int const by_regs = regs_sm / std::max(1, ((m == kPlain ? fp : fa).numRegs + 7) / 8 * 8 * 128);
        g_conv_per_sm[m] = std::max(1, std::min(std::min(by_smem, by_regs), 8));
    }
    SIL_CUDA_CHECK(cudaFuncSetAttribute(wgrad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        static_cast<int>(wgrad_smem())));
    void const* const walk_fns[kWalkKinds] = {
        reinterpret_cast<void const*>(inc_forward_kernel), reinterpret_cast<void const*>(out_forward_kernel),
        reinterpret_cast<void const*>(out_gather_kernel),  reinterpret_cast<void const*>(pool_kernel),
        reinterpret_cast<void const*>(copy_act_kernel),    reinterpret_cast<void const*>(features_kernel),
        reinterpret_cast<void const*>(wrap_pre_kernel),    reinterpret_cast<void const*>(wrap_post_kernel),
        reinterpret_cast<void const*>(lognu_feature_kernel), reinterpret_cast<void const*>(wrap_e2_kernel),
        reinterpret_cast<void const*>(upadd_kernel)};
    for (int k = 0; k < kWalkKinds; ++k) {
        cudaFuncAttributes a {};
        SIL_CUDA_CHECK(cudaFuncGetAttributes(&a, walk_fns[k]));
        int const regs = (a.numRegs + 7) / 8 * 8;   // per-thread allocation granularity
        int const by_regs = regs_sm / std::max(1, regs * 256);
        int const by_smem = smem_sm / static_cast<int>(a.sharedSizeBytes + 1024);
        g_walk_per_sm[k] = std::max(1, std::min(std::min(by_regs, by_smem), 8));
    }
    g_attr_done = true;
    return SIL_OK;
}

// Persistent grid: every CTA resident in one wave (a second wave would
// serialise behind the first).
int conv_grid(int ntiles, int mode)
{
    int const per_sm = g_conv_per_sm[mode] > 0 ? g_conv_per_sm[mode] : 1;
    return std::max(1, std::min(ntiles, per_sm * (g_sms > 0 ? g_sms : 148)));
}

// Blocks of 256 threads for a grid-stride kernel: four resident waves (its
// blocks per multiprocessor from registers and shared memory), so blocks
// that finish early pick up the remaining work; fewer when the work is
// smaller.
unsigned walk_grid(Table const& t, int per, int kind)
{
    int64_t const chunks = (t.px_base[t.nimg] * per + 255) / 256;
    int64_t const wave = 4 * static_cast<int64_t>(g_walk_per_sm[kind]) * (g_sms > 0 ? g_sms : 148);
    return static_cast<unsigned>(std::max<int64_t>(1, std::min<int64_t>(chunks, wave)));
}

unsigned item_grid(int nitems, int kind)
{
    return static_cast<unsigned>(std::max(1, std::min(nitems, 4 * g_walk_per_sm[kind] * (g_sms > 0 ? g_sms : 148))));
}


// Launch of a kernel that calls after_previous.
template <class... P, class... A>
cudaError_t launch_after(void (*kernel)(P...), dim3 grid, unsigned block, size_t smem, cudaStream_t st, A const&... args)
{
    cudaLaunchAttribute early {};
    early.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    early.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &early;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
}

// 1024-byte aligned dynamic shared memory: the kernels index from the start
// of the dynamic block, which the runtime aligns to at least 1024 bytes when
// the kernel declares it so.
sil_status launch_conv(cudaStream_t st, Table const& t, int mode, bf16 const* in, bf16 const* in2, float const* gin,
                       bf16 const* w, float const* bias, int relu, bf16* out, float* out_f32, int accumulate,
                       int* err, float* out_taps = nullptr, float const* wout = nullptr, int64_t taps_stride = 0)
{
    if (t.nimg == 0 || t.tile_base[t.nimg] == 0) return SIL_OK;
    ConvOut const dst {bias, relu, out, out_f32, accumulate, out_taps, taps_stride};
    int const grid = conv_grid(t.tile_base[t.nimg], mode);
    if (mode == kPlain) SIL_CUDA_CHECK(launch_after(conv3x3_plain_kernel, grid, 128, conv_smem(mode), st, t, in, w,
                                                    dst, wout, err));
    else SIL_CUDA_CHECK(launch_after(conv3x3_kernel, grid, 128, conv_smem(mode), st, t, mode, in, in2, gin, w, dst,
                                     err));
    SIL_CUDA_CHECK(cudaGetLastError());
    return SIL_OK;
}

template <class K>
dim3 image_grid(Table const& t, int per_px, K)
{
    int64_t maxpx = 0;
    for (int k = 0; k < t.nimg; ++k) maxpx = std::max<int64_t>(maxpx, static_cast<int64_t>(t.img[k].h + 2) * (t.img[k].w + 2));
    return dim3(static_cast<unsigned>((maxpx * per_px + 255) / 256), static_cast<unsigned>(t.nimg));
}

} // namespace

Net::Net() = default;

Net::~Net()
{
    cudaFree(params);
    cudaFree(grad);
    cudaFree(adam_m);
    cudaFree(adam_v);
    cudaFree(wbf);
    cudaFree(wbf_t);
    cudaFree(error_flag);
}

sil_status Net::init(uint64_t seed, cudaStream_t stream)
{
    if (params == nullptr) {
        SIL_CUDA_CHECK(cudaMalloc(&params, sizeof(float) * kNumParams));
        SIL_CUDA_CHECK(cudaMalloc(&grad, sizeof(float) * kNumParams));
        SIL_CUDA_CHECK(cudaMalloc(&adam_m, sizeof(float) * kNumParams));
        SIL_CUDA_CHECK(cudaMalloc(&adam_v, sizeof(float) * kNumParams));
        SIL_CUDA_CHECK(cudaMalloc(&wbf, sizeof(bf16) * kNumBig * kBigW));
        SIL_CUDA_CHECK(cudaMalloc(&wbf_t, sizeof(bf16) * kNumBig * kBigW));
        SIL_CUDA_CHECK(cudaMalloc(&error_flag, sizeof(int)));
        SIL_CUDA_CHECK(cudaMemsetAsync(error_flag, 0, sizeof(int), stream));
    }
    // He-normal weights, zero biases (host RNG, reproducible per seed).
    std::vector<float> h(kNumParams, 0.0f);
    std::mt19937_64 rng(seed);
    auto fill = [&](int off, int count, int fan_in) {
        std::normal_distribution<float> nd(0.0f, std::sqrt(2.0f / static_cast<float>(fan_in)));
        for (int i = 0; i < count; ++i) h[off + i] = nd(rng);
    };
    fill(kOffIn, kInW, kTaps * 2);
    for (int j = 0; j < kNumBig; ++j) fill(kOffBig + j * kBigParams, kBigW, kTaps * kCh);
    fill(kOffOut, kOutW, kTaps * kCh);
    for (int i = 0; i < kOutW; ++i) h[kOffOut + i] *= 0.5f;
    return set_params(h.data(), stream);
}

sil_status Net::set_params(float const* host, cudaStream_t stream)
{
    if (params == nullptr) {
        sil_status const st = init(0, stream);
        if (st != SIL_OK) return st;
    }
    SIL_CUDA_CHECK(cudaMemcpyAsync(params, host, sizeof(float) * kNumParams, cudaMemcpyHostToDevice, stream));
    SIL_CUDA_CHECK(cudaMemsetAsync(adam_m, 0, sizeof(float) * kNumParams, stream));
    SIL_CUDA_CHECK(cudaMemsetAsync(adam_v, 0, sizeof(float) * kNumParams, stream));
    adam_t = 0;
    return refresh(stream);
}

sil_status Net::get_params(float* host, cudaStream_t stream)
{
    SIL_CUDA_CHECK(cudaMemcpyAsync(host, params, sizeof(float) * kNumParams, cudaMemcpyDeviceToHost, stream));
    SIL_CUDA_CHECK(cudaStreamSynchronize(stream));
    return SIL_OK;
}

sil_status Net::refresh(cudaStream_t stream)
{
    int const n = kNumBig * kBigW;
    convert_weights_kernel<<<(n + 255) / 256, 256, 0, stream>>>(params, static_cast<bf16*>(wbf), static_cast<bf16*>(wbf_t));
    SIL_CUDA_CHECK(cudaGetLastError());
    return SIL_OK;
}

Workspace* Net::workspace(std::vector<Sample> const& samples, cudaStream_t stream, sil_status* st)
{
    (void)stream;
    for (auto& w : cache_) {
        if (w->samples.size() != samples.size()) continue;
        bool same = true;
        for (size_t i = 0; i < samples.size() && same; ++i)
            same = w->samples[i].nx == samples[i].nx && w->samples[i].ny == samples[i].ny
                   && w->samples[i].offset == samples[i].offset;
        if (same) {
            *st = SIL_OK;
            return w.get();
        }
    }
    if (cache_.size() >= 4) cache_.erase(cache_.begin());
    auto w = std::make_unique<Workspace>();
    *st = w->build(samples);
    if (*st != SIL_OK) return nullptr;
    cache_.push_back(std::move(w));
    return cache_.back().get();
}

namespace {

bf16 const* big_w(Net const& net, int kind, int wl) { return static_cast<bf16 const*>(net.wbf) + big_index(kind, wl) * kBigW; }
bf16 const* big_wt(Net const& net, int kind, int wl) { return static_cast<bf16 const*>(net.wbf_t) + big_index(kind, wl) * kBigW; }
float const* big_b(Net const& net, int kind, int wl) { return net.params + kOffBig + big_index(kind, wl) * kBigParams + kBigW; }
float* big_grad(Net& net, int kind, int wl) { return net.grad + kOffBig + big_index(kind, wl) * kBigParams; }
int weight_level_enc(int l) { return std::min(l - 1, 2); }   // encoder convs of level l >= 1
int weight_level_dec(int l) { return std::min(l, 2); }       // decoder conv producing level l

dim3 node_grid(Workspace const& w)
{
    return dim3(static_cast<unsigned>((w.max_node_per_sample + 255) / 256), static_cast<unsigned>(w.samples.size()));
}

dim3 top_grid(Workspace const& w)
{
    int64_t m = 0;
    for (Img const& i : w.levels[0].img) m = std::max<int64_t>(m, static_cast<int64_t>(i.h + 2) * (i.w + 2));
    return dim3(static_cast<unsigned>((m + 255) / 256), static_cast<unsigned>(w.samples.size()));
}

sil_status dots(Workspace& w, cudaStream_t st, int set, float const* a1, float const* b1, float const* a2,
                float const* b2, float const* a3, float const* b3)
{
    int const n = static_cast<int>(w.samples.size());
    dots_kernel<<<dim3(w.dot_blocks, n), kDotBlock, 0, st>>>(w.ss, a1, b1, a2, b2, a3, b3, w.dparts.as<double>(),
                                                             w.dot_blocks);
    dots_finish_kernel<<<1, std::max(32, ((3 * n + 31) / 32) * 32), 0, st>>>(w.dparts.as<double>(), n, w.dot_blocks,
                                                                            w.dots.as<double>() + set * 3 * n);
    SIL_CUDA_CHECK(cudaGetLastError());
    return SIL_OK;
}

Table deepest_table(Workspace const& w, int l);
Table dec_table(Workspace const& w, int l);

// Network forward on the feature image in w.feat; result in w.unet.  With
// `keep` every activation the backward pass reads is stored; without it the
// output convolution is folded into the last decoder convolution.
sil_status net_forward(Net& net, Workspace& w, cudaStream_t st, bool keep)
{
    int const D = static_cast<int>(w.levels.size());
    int* err = net.error_flag;
    {
        Table const t = w.table(0, -1, false);
        SIL_CUDA_CHECK(launch_after(inc_forward_kernel, walk_grid(t, 1, kWalkInc), 256, 0, st, t, w.feat.as<float>(),
                                    net.params, w.h[0].as<bf16>()));
        SIL_CUDA_CHECK(cudaGetLastError());
    }
    for (int l = 1; l < D; ++l) {
        int const wl = weight_level_enc(l);
        Table const t = w.table(l, l - 1, true);
        SIL_CUDA_CHECK(launch_after(pool_kernel, walk_grid(t, kChunks, kWalkPool), 256, 0, st, t,
                                    w.h[l - 1].as<bf16>(), w.pin[l].as<bf16>()));
        SIL_CUDA_CHECK(cudaGetLastError());
        Table const t2 = w.table(l, -1, false);
        sil_status s = launch_conv(st, t2, kPlain, w.pin[l].as<bf16>(), nullptr, nullptr, big_w(net, kDown, wl),
                                   big_b(net, kDown, wl), 1, w.p[l].as<bf16>(), nullptr, 0, err);
        if (s != SIL_OK) return s;
        s = launch_conv(st, t2, kPlain, w.p[l].as<bf16>(), nullptr, nullptr, big_w(net, kEnc, wl), big_b(net, kEnc, wl),
                        1, w.h[l].as<bf16>(), nullptr, 0, err);
        if (s != SIL_OK) return s;
    }
    // g at each image's deepest level is its h.
    for (int l = 0; l < D; ++l) {
        Table const t = deepest_table(w, l);
        if (t.nimg == 0) continue;
        copy_act_kernel<<<walk_grid(t, kChunks, kWalkCopy), 256, 0, st>>>(t, w.h[l].as<bf16>(), w.g[l].as<bf16>());
        SIL_CUDA_CHECK(cudaGetLastError());
    }
    int64_t const top = w.levels[0].npx;
    for (int l = D - 2; l >= 0; --l) {
        int const wl = weight_level_dec(l);
        Table const tt = dec_table(w, l);
        if (tt.nimg == 0) continue;
        bool const fold = l == 0 && !keep;
        sil_status s;
        if (keep) {
            s = launch_conv(st, tt, kUpAdd, w.h[l].as<bf16>(), w.g[l + 1].as<bf16>(), nullptr, big_w(net, kDec, wl),
                            big_b(net, kDec, wl), 1, w.g[l].as<bf16>(), nullptr, 0, err);
        } else {
            // the pooled input of this level (pin) has been consumed by the encoder: it holds the sum
            SIL_CUDA_CHECK(launch_after(upadd_kernel, walk_grid(tt, kChunks, kWalkUpAdd), 256, 0, st, tt,
                                        w.h[l].as<bf16>(), w.g[l + 1].as<bf16>(), w.pin[l].as<bf16>()));
            SIL_CUDA_CHECK(cudaGetLastError());
            s = launch_conv(st, tt, kPlain, w.pin[l].as<bf16>(), nullptr, nullptr, big_w(net, kDec, wl),
                            big_b(net, kDec, wl), 1, fold ? nullptr : w.g[l].as<bf16>(), nullptr, 0, err,
                            fold ? w.taps.as<float>() : nullptr, net.params + kOffOut, top);
        }
        if (s != SIL_OK) return s;
    }
    if (keep) {
        Table const t = w.table(0, -1, false);
        SIL_CUDA_CHECK(launch_after(out_forward_kernel, walk_grid(t, 1, kWalkOut), 256, 0, st, t, w.g[0].as<bf16>(),
                                    net.params, w.unet.as<float>()));
    } else {
        Table const td = dec_table(w, 0);
        if (td.nimg > 0)
            SIL_CUDA_CHECK(launch_after(out_gather_kernel, walk_grid(td, 1, kWalkGather), 256, 0, st, td,
                                        w.taps.as<float>(), top, net.params, w.unet.as<float>()));
        Table const t1 = deepest_table(w, 0);  // single-level images: no decoder
        if (t1.nimg > 0)
            SIL_CUDA_CHECK(launch_after(out_forward_kernel, walk_grid(t1, 1, kWalkOut), 256, 0, st, t1,
                                        w.g[0].as<bf16>(), net.params, w.unet.as<float>()));
    }
    SIL_CUDA_CHECK(cudaGetLastError());
    return SIL_OK;
}

// Images of level l that have level l+1 (the decoder's images).
Table dec_table(Workspace const& w, int l)
{
    Table t = w.table(l, l + 1, false);
    Table tt {};
    tt.active = t.active;
    tt.tile_base[0] = 0;
    for (int k = 0; k < t.nimg; ++k) {
        if (t.aux[k].h == 0) continue;
        int const q = tt.nimg++;
        tt.img[q] = t.img[k];
        tt.aux[q] = t.aux[k];
        tt.sample[q] = t.sample[k];
        tt.px_base[q + 1] = tt.px_base[q] + static_cast<int64_t>(t.img[k].h + 2) * (t.img[k].w + 2);
        tt.tile_base[q + 1] = tt.tile_base[q] + (t.tile_base[k + 1] - t.tile_base[k]);
    }
    return tt;
}

// Images whose deepest level is l.
Table deepest_table(Workspace const& w, int l)
{
    Table t {};
    t.active = w.active;
    Level const& L = w.levels[l];
    for (size_t k = 0; k < L.images.size(); ++k) {
        if (w.depth[L.images[k]] - 1 != l) continue;
        int const q = t.nimg++;
        t.img[q] = L.img[k];
        t.aux[q] = L.img[k];
        t.sample[q] = L.images[k];
        t.px_base[q + 1] = t.px_base[q] + static_cast<int64_t>(L.img[k].h + 2) * (L.img[k].w + 2);
        t.tile_base[q + 1] = t.tile_base[q];
    }
    return t;
}

sil_status wgrad(Net& net, Workspace& w, cudaStream_t st, Table const& t, int mode, bf16 const* in, bf16 const* in2,
                 float const* dy, bf16 const* y, float* grad_out)
{
    if (t.nimg == 0 || t.tile_base[t.nimg] == 0) return SIL_OK;
    int const grid = std::min(w.wgrad_grid, t.tile_base[t.nimg]);
    SIL_CUDA_CHECK(launch_after(wgrad_kernel, grid, 128, wgrad_smem(), st, t, mode, in, in2, dy, y,
                                w.wparts.as<float>(), net.error_flag));
    SIL_CUDA_CHECK(launch_after(reduce_parts_kernel, (kWgradParts + 31) / 32, 256, 0, st, w.wparts.as<float>(), grid,
                                kWgradParts, grad_out));
    SIL_CUDA_CHECK(cudaGetLastError());
    return SIL_OK;
}

// Network backward from the gradient in w.gnet: accumulates into net.grad.
sil_status net_backward(Net& net, Workspace& w, cudaStream_t st)
{
    int const D = static_cast<int>(w.levels.size());
    int* err = net.error_flag;
    for (int l = 0; l < D; ++l) {
        size_t const a = static_cast<size_t>(w.levels[l].npx) * kCh * sizeof(float);
        SIL_CUDA_CHECK(cudaMemsetAsync(w.dh[l].p, 0, a, st));
        SIL_CUDA_CHECK(cudaMemsetAsync(w.dg[l].p, 0, a, st));
    }
    Table const t0 = w.table(0, -1, false);
    int const thin_blocks = std::min(w.thin_grid, t0.tile_base[t0.nimg]);
    // output convolution
    SIL_CUDA_CHECK(launch_after(out_backward_data_kernel, image_grid(t0, 1, 0), 256, 0, st, t0, w.gnet.as<float>(),
                                net.params, w.dg[0].as<float>()));
    SIL_CUDA_CHECK(launch_after(out_wgrad_kernel, thin_blocks, kThinBlock, 0, st, t0, w.gnet.as<float>(),
                                w.g[0].as<bf16>(), w.wparts.as<float>()));
    SIL_CUDA_CHECK(launch_after(reduce_parts_kernel, (kOutW + 1 + 31) / 32, 256, 0, st, w.wparts.as<float>(),
                                thin_blocks, kOutW + 1, net.grad + kOffOut));
    SIL_CUDA_CHECK(cudaGetLastError());
    // decoder, top-down
    for (int l = 0; l <= D - 2; ++l) {
        int const wl = weight_level_dec(l);
        Table const t = dec_table(w, l);
        if (t.nimg == 0) continue;
        sil_status s = wgrad(net, w, st, t, kUpAdd, w.h[l].as<bf16>(), w.g[l + 1].as<bf16>(), w.dg[l].as<float>(),
                             w.g[l].as<bf16>(), big_grad(net, kDec, wl));
        if (s != SIL_OK) return s;
        s = launch_conv(st, t, kMasked, w.g[l].as<bf16>(), w.g[l].as<bf16>(), w.dg[l].as<float>(), big_wt(net, kDec, wl),
                        nullptr, 0, nullptr, w.dx[l].as<float>(), 0, err);
        if (s != SIL_OK) return s;
        SIL_CUDA_CHECK(launch_after(upadd_adjoint_skip_kernel, image_grid(t, 8, 0), 256, 0, st, t, w.dx[l].as<float>(),
                                    w.dh[l].as<float>()));
        // coarse part: table over level l+1 with aux = level l
        Table tc {};
        tc.nimg = t.nimg;
        for (int k = 0; k < t.nimg; ++k) {
            tc.img[k] = t.aux[k];
            tc.aux[k] = t.img[k];
        }
        SIL_CUDA_CHECK(launch_after(upadd_adjoint_coarse_kernel, image_grid(tc, 8, 0), 256, 0, st, tc,
                                    w.dx[l].as<float>(), w.dg[l + 1].as<float>()));
        SIL_CUDA_CHECK(cudaGetLastError());
    }
    // deepest level of each image: g = h
    for (int l = 0; l < D; ++l) {
        Table const t = deepest_table(w, l);
        if (t.nimg == 0) continue;
        SIL_CUDA_CHECK(launch_after(upadd_adjoint_skip_kernel, image_grid(t, 8, 0), 256, 0, st, t, w.dg[l].as<float>(),
                                    w.dh[l].as<float>()));
        SIL_CUDA_CHECK(cudaGetLastError());
    }
    // encoder, bottom-up
    for (int l = D - 1; l >= 1; --l) {
        int const wl = weight_level_enc(l);
        Table const t = w.table(l, -1, false);
        sil_status s = wgrad(net, w, st, t, kPlain, w.p[l].as<bf16>(), nullptr, w.dh[l].as<float>(), w.h[l].as<bf16>(),
                             big_grad(net, kEnc, wl));
        if (s != SIL_OK) return s;
        s = launch_conv(st, t, kMasked, w.h[l].as<bf16>(), w.h[l].as<bf16>(), w.dh[l].as<float>(), big_wt(net, kEnc, wl),
                        nullptr, 0, nullptr, w.dx[l].as<float>(), 0, err);
        if (s != SIL_OK) return s;
        Table const tp = w.table(l, l - 1, true);
        s = wgrad(net, w, st, t, kPlain, w.pin[l].as<bf16>(), nullptr, w.dx[l].as<float>(), w.p[l].as<bf16>(),
                  big_grad(net, kDown, wl));
        if (s != SIL_OK) return s;
        // data gradient of the down convolution into dg[l] (scratch), then pool adjoint into dh[l-1]
        s = launch_conv(st, t, kMasked, w.p[l].as<bf16>(), w.p[l].as<bf16>(), w.dx[l].as<float>(),
                        big_wt(net, kDown, wl), nullptr, 0, nullptr, w.dg[l].as<float>(), 0, err);
        if (s != SIL_OK) return s;
        Table tf {};
        tf.nimg = tp.nimg;
        for (int k = 0; k < tp.nimg; ++k) {
            tf.img[k] = tp.aux[k];   // fine level l-1
            tf.aux[k] = tp.img[k];   // coarse level l
        }
        SIL_CUDA_CHECK(launch_after(pool_adjoint_kernel, image_grid(tf, 8, 0), 256, 0, st, tf, w.dg[l].as<float>(),
                                    w.dh[l - 1].as<float>()));
        SIL_CUDA_CHECK(cudaGetLastError());
    }
    // input convolution
    SIL_CUDA_CHECK(launch_after(inc_wgrad_kernel, thin_blocks, kThinBlock, 0, st, t0, w.dh[0].as<float>(),
                                w.h[0].as<bf16>(), w.feat.as<float>(), w.wparts.as<float>()));
    SIL_CUDA_CHECK(launch_after(reduce_parts_kernel, (kInW + kCh + 31) / 32, 256, 0, st, w.wparts.as<float>(),
                                thin_blocks, kInW + kCh, net.grad + kOffIn));
    SIL_CUDA_CHECK(cudaGetLastError());
    return SIL_OK;
}

// Preconditioner forward: out = M(b) for the batch of w (nu per node).
// dinv: the inverse operator diagonal, or NULL to compute it here.
sil_status precond_forward(Net& net, Workspace& w, float const* nu, float const* dinv, float const* b, float* out,
                           cudaStream_t st, bool keep = false, int const* active = nullptr)
{
    w.active = active;
    w.ss.active = active;
    if (dinv == nullptr) {
        dinv_kernel<<<static_cast<unsigned>(w.nwitems), 256, 0, st>>>(w.ss, w.witems.as<WrapItem>(), nu, w.dinv.as<float>());
        dinv = w.dinv.as<float>();
    }
    WrapItem const* items = w.witems.as<WrapItem>();
    Table const t0 = w.table(0, -1, false);
    wrap_pre_kernel<<<item_grid(w.nstrips, kWalkPre), 256, 0, st>>>(w.ss, nu, dinv, b, w.r1.as<float>(),
                                                                    w.wpart.as<double>());
    SIL_CUDA_CHECK(launch_after(wrap_finish_kernel, static_cast<unsigned>(w.samples.size()), 32, 0, st, w.ss,
                                w.wpart.as<double>(), w.dots.as<double>()));
    SIL_CUDA_CHECK(cudaGetLastError());
    float const* lognu = (w.lognu_for != nullptr && w.lognu_for == nu) ? w.lognu.as<float>() : nullptr;
    SIL_CUDA_CHECK(launch_after(features_kernel, walk_grid(t0, 1, kWalkFeat), 256, 0, st, w.ss, t0, w.r1.as<float>(),
                                nu, dinv, w.dots.as<double>(), lognu, w.feat.as<float>()));
    SIL_CUDA_CHECK(cudaGetLastError());
    sil_status s = net_forward(net, w, st, keep);
    if (s != SIL_OK) return s;
    SIL_CUDA_CHECK(launch_after(wrap_e2_kernel, item_grid(w.nwitems, kWalkE2), 256, 0, st, w.ss, items, dinv, b,
                                w.unet.as<float>(), w.dots.as<double>(), w.e2.as<float>()));
    SIL_CUDA_CHECK(launch_after(wrap_post_kernel, item_grid(w.nstrips, kWalkPost), 256, 0, st, w.ss, nu, dinv, b,
                                w.e2.as<float>(), out));
    SIL_CUDA_CHECK(cudaGetLastError());
    return SIL_OK;
}

sil_status check_samples(std::vector<Sample> const& samples)
{
    if (samples.empty() || samples.size() > kMaxImages) return fail(SIL_ERR_INVALID, "precond: 1 to 64 samples per batch");
    for (Sample const& s : samples)
        if (s.nx < 3 || s.ny < 3 || s.offset < 0) return fail(SIL_ERR_INVALID, "precond: bad sample geometry");
    return SIL_OK;
}

} // namespace

sil_status Net::apply(std::vector<Sample> const& samples, float const* nu, float const* r, float* out, cudaStream_t stream,
                      int const* active)
{
    if (sil_status s = check_samples(samples); s != SIL_OK) return s;
    if (sil_status s = ensure_attributes(); s != SIL_OK) return s;
    sil_status st = SIL_OK;
    Workspace* w = workspace(samples, stream, &st);
    if (w == nullptr) return st;
    return precond_forward(*this, *w, nu, nullptr, r, out, stream, false, active);
}

sil_status Net::prepare(std::vector<Sample> const& samples, cudaStream_t stream, Workspace** out)
{
    if (sil_status s = check_samples(samples); s != SIL_OK) return s;
    if (sil_status s = ensure_attributes(); s != SIL_OK) return s;
    sil_status st = SIL_OK;
    *out = workspace(samples, stream, &st);
    return *out == nullptr ? st : SIL_OK;
}

sil_status Net::set_static_nu(Workspace* w, float const* nu, cudaStream_t stream)
{
    w->lognu_for = nullptr;
    if (nu == nullptr) return SIL_OK;
    if (w->lognu.p == nullptr) {
        if (sil_status st = w->lognu.alloc(sizeof(float) * w->levels[0].npx); st != SIL_OK) return st;
    }
    w->active = nullptr;
    w->ss.active = nullptr;
    Table const t0 = w->table(0, -1, false);
    lognu_feature_kernel<<<walk_grid(t0, 1, kWalkLogNu), 256, 0, stream>>>(w->ss, t0, nu, w->lognu.as<float>());
    SIL_CUDA_CHECK(cudaGetLastError());
    w->lognu_for = nu;
    return SIL_OK;
}

sil_status Net::forward(Workspace* w, float const* nu, float const* dinv, float const* r, float* out,
                        cudaStream_t stream, int const* active)
{
    return precond_forward(*this, *w, nu, dinv, r, out, stream, false, active);
}

sil_status Net::loss_grad(std::vector<Sample> const& samples, float const* nu, float const* b, float const* x,
                          double* loss, std::vector<double>* per_sample, cudaStream_t stream)
{
    if (sil_status s = check_samples(samples); s != SIL_OK) return s;
    if (sil_status s = ensure_attributes(); s != SIL_OK) return s;
    sil_status st = SIL_OK;
    Workspace* w = workspace(samples, stream, &st);
    if (w == nullptr) return st;
    int const n = static_cast<int>(samples.size());
    SIL_CUDA_CHECK(cudaMemsetAsync(grad, 0, sizeof(float) * kNumParams, stream));
    st = precond_forward(*this, *w, nu, nullptr, b, w->u.as<float>(), stream, true);
    if (st != SIL_OK) return st;
    dim3 const ng = node_grid(*w);
    float const* fnu = nu;
    kapply_kernel<<<ng, 256, 0, stream>>>(w->ss, fnu, w->u.as<float>(), w->ku.as<float>());
    SIL_CUDA_CHECK(cudaGetLastError());
    // set 1: u.b, u.Ku ; set 2: x.b
    if (sil_status s = dots(*w, stream, 1, w->u.as<float>(), b, w->u.as<float>(), w->ku.as<float>(), nullptr, nullptr);
        s != SIL_OK)
        return s;
    if (sil_status s = dots(*w, stream, 2, x, b, nullptr, nullptr, nullptr, nullptr); s != SIL_OK) return s;
    double const* d = w->dots.as<double>();
    loss_grad_u_kernel<<<ng, 256, 0, stream>>>(w->ss, b, w->ku.as<float>(), d + 3 * n, d + 6 * n, w->gu.as<float>());
    // g_e2 = g_u - w K (dinv g_u)
    jacobi_kernel<<<ng, 256, 0, stream>>>(w->ss, fnu, w->dinv.as<float>(), w->gu.as<float>(), nullptr, nullptr, 1.0f,
                                          w->tmp.as<float>());
    kapply_kernel<<<ng, 256, 0, stream>>>(w->ss, fnu, w->tmp.as<float>(), w->ge2.as<float>());
    axpby_kernel<<<ng, 256, 0, stream>>>(w->ss, 1.0f, w->gu.as<float>(), -kOmega, w->ge2.as<float>(), w->ge2.as<float>());
    net_grad_kernel<<<top_grid(*w), 256, 0, stream>>>(w->ss, w->ge2.as<float>(), w->dinv.as<float>(), d,
                                                      w->gnet.as<float>());
    SIL_CUDA_CHECK(cudaGetLastError());
    st = net_backward(*this, *w, stream);
    if (st != SIL_OK) return st;
    std::vector<double> hd(9 * n);
    SIL_CUDA_CHECK(cudaMemcpyAsync(hd.data(), d, sizeof(double) * 9 * n, cudaMemcpyDeviceToHost, stream));
    int herr = 0;
    SIL_CUDA_CHECK(cudaMemcpyAsync(&herr, error_flag, sizeof(int), cudaMemcpyDeviceToHost, stream));
    SIL_CUDA_CHECK(cudaStreamSynchronize(stream));
    if (herr != 0) return fail(SIL_ERR_BUDGET, "precond: a tensor-core wait ran out of its bound");
    double total = 0.0;
    if (per_sample != nullptr) per_sample->assign(n, 0.0);
    for (int i = 0; i < n; ++i) {
        double const ub = hd[3 * n + 3 * i], uku = hd[3 * n + 3 * i + 1], xb = hd[6 * n + 3 * i];
        double const li = (uku > 0 && xb > 0) ? 1.0 - ub * ub / (uku * xb) : 1.0;
        total += li;
        if (per_sample != nullptr) (*per_sample)[i] = li;
    }
    *loss = total / n;
    return SIL_OK;
}

sil_status Net::adam_step(float lr, cudaStream_t stream)
{
    ++adam_t;
    float const b1t = 1.0f - std::pow(0.9f, static_cast<float>(adam_t));
    float const b2t = 1.0f - std::pow(0.999f, static_cast<float>(adam_t));
    adam_kernel<<<(kNumParams + 255) / 256, 256, 0, stream>>>(params, grad, adam_m, adam_v, kNumParams, lr, b1t, b2t);
    SIL_CUDA_CHECK(cudaGetLastError());
    return refresh(stream);
}

sil_status Net::debug_fetch(int which, int level, float* host, int64_t count, cudaStream_t stream)
{
    if (cache_.empty()) return fail(SIL_ERR_INVALID, "precond: no workspace yet");
    Workspace& w = *cache_.back();
    if (level < 0 || level >= static_cast<int>(w.levels.size())) return fail(SIL_ERR_INVALID, "precond: bad level");
    int64_t const n = w.levels[level].npx * kCh;
    std::vector<uint16_t> tmp;
    auto get_bf = [&](DevBuf const& b) -> sil_status {
        if (count < n) return fail(SIL_ERR_INVALID, "precond: host buffer too small");
        tmp.resize(n);
        SIL_CUDA_CHECK(cudaMemcpyAsync(tmp.data(), b.p, n * 2, cudaMemcpyDeviceToHost, stream));
        SIL_CUDA_CHECK(cudaStreamSynchronize(stream));
        for (int64_t i = 0; i < n; ++i) {
            uint32_t const u = static_cast<uint32_t>(tmp[i]) << 16;
            std::memcpy(host + i, &u, 4);
        }
        return SIL_OK;
    };
    auto get_f = [&](void const* p, int64_t m) -> sil_status {
        if (count < m) return fail(SIL_ERR_INVALID, "precond: host buffer too small");
        SIL_CUDA_CHECK(cudaMemcpyAsync(host, p, m * 4, cudaMemcpyDeviceToHost, stream));
        SIL_CUDA_CHECK(cudaStreamSynchronize(stream));
        return SIL_OK;
    };
    switch (which) {
    case 0: return get_bf(w.h[level]);
    case 1: return get_bf(w.p[level]);
    case 2: return get_bf(w.g[level]);
    case 3: return get_f(w.dh[level].p, n);
    case 4: return get_f(w.dg[level].p, n);
    case 5: return get_f(w.feat.p, w.levels[0].npx * 2);
    case 6: return get_f(w.unet.p, w.levels[0].npx);
    case 7: return get_f(w.u.p, w.nodes);
    case 8: return get_f(w.gnet.p, w.levels[0].npx);
    default: return fail(SIL_ERR_INVALID, "precond: unknown debug tensor");
    }
}

} // namespace nn
} // namespace sil

// ------------------------------------------------------------------ C API

using sil::nn::Sample;

namespace {

sil_status to_samples(sil_precond_sample const* in, int n, std::vector<Sample>* out)
{
    if (in == nullptr || n < 1 || n > sil::nn::kMaxImages) return sil::fail(SIL_ERR_INVALID, "precond: 1 to 64 samples");
    out->resize(n);
    for (int i = 0; i < n; ++i) (*out)[i] = {in[i].nx, in[i].ny, in[i].offset};
    return SIL_OK;
}

} // namespace

extern "C" {

int64_t sil_precond_num_params(void) { return sil::nn::kNumParams; }

sil_status sil_precond_create(sil_precond* out, uint64_t seed, sil_stream stream)
{
    if (out == nullptr) return sil::fail(SIL_ERR_INVALID, "sil_precond_create: NULL");
    auto* p = new (std::nothrow) sil_precond_s;
    if (p == nullptr) return sil::fail(SIL_ERR_ALLOC, "sil_precond_create");
    sil_status const st = p->net.init(seed, static_cast<cudaStream_t>(stream));
    if (st != SIL_OK) {
        delete p;
        return st;
    }
    *out = p;
    return SIL_OK;
}

void sil_precond_destroy(sil_precond p) { delete p; }

sil_status sil_precond_get_params(sil_precond p, float* host)
{
    if (p == nullptr || host == nullptr) return sil::fail(SIL_ERR_INVALID, "sil_precond_get_params: NULL");
    return p->net.get_params(host, nullptr);
}

sil_status sil_precond_set_params(sil_precond p, const float* host, sil_stream stream)
{
    if (p == nullptr || host == nullptr) return sil::fail(SIL_ERR_INVALID, "sil_precond_set_params: NULL");
    return p->net.set_params(host, static_cast<cudaStream_t>(stream));
}

sil_status sil_precond_get_optimizer_state(sil_precond p, float* m, float* v, int64_t* step)
{
    if (p == nullptr) return sil::fail(SIL_ERR_INVALID, "sil_precond_get_optimizer_state: NULL");
    sil::nn::Net& net = p->net;
    size_t const bytes = sizeof(float) * sil::nn::kNumParams;
    if (net.adam_m == nullptr) {
        if (m != nullptr) std::memset(m, 0, bytes);
        if (v != nullptr) std::memset(v, 0, bytes);
        if (step != nullptr) *step = 0;
        return SIL_OK;
    }
    SIL_CUDA_CHECK(cudaDeviceSynchronize());
    if (m != nullptr) SIL_CUDA_CHECK(cudaMemcpy(m, net.adam_m, bytes, cudaMemcpyDeviceToHost));
    if (v != nullptr) SIL_CUDA_CHECK(cudaMemcpy(v, net.adam_v, bytes, cudaMemcpyDeviceToHost));
    if (step != nullptr) *step = net.adam_t;
    return SIL_OK;
}

sil_status sil_precond_set_optimizer_state(sil_precond p, const float* m, const float* v, int64_t step,
                                           sil_stream stream)
{
    if (p == nullptr || m == nullptr || v == nullptr || step < 0 || step > (int64_t(1) << 30))
        return sil::fail(SIL_ERR_INVALID, "sil_precond_set_optimizer_state: NULL state or bad step");
    sil::nn::Net& net = p->net;
    if (net.adam_m == nullptr) return sil::fail(SIL_ERR_INVALID, "sil_precond_set_optimizer_state: set the parameters first");
    cudaStream_t const s = static_cast<cudaStream_t>(stream);
    size_t const bytes = sizeof(float) * sil::nn::kNumParams;
    SIL_CUDA_CHECK(cudaMemcpyAsync(net.adam_m, m, bytes, cudaMemcpyHostToDevice, s));
    SIL_CUDA_CHECK(cudaMemcpyAsync(net.adam_v, v, bytes, cudaMemcpyHostToDevice, s));
    SIL_CUDA_CHECK(cudaStreamSynchronize(s));
    net.adam_t = static_cast<int>(step);
    return SIL_OK;
}

sil_status sil_precond_apply(sil_precond p, sil_stream stream, const sil_precond_sample* samples, int n,
                             const float* nu, const float* r, float* out)
{
    if (p == nullptr || nu == nullptr || r == nullptr || out == nullptr)
        return sil::fail(SIL_ERR_INVALID, "sil_precond_apply: NULL");
    std::vector<Sample> s;
    if (sil_status st = to_samples(samples, n, &s); st != SIL_OK) return st;
    return p->net.apply(s, nu, r, out, static_cast<cudaStream_t>(stream));
}

sil_status sil_precond_apply_active(sil_precond p, sil_stream stream, const sil_precond_sample* samples, int n,
                                    const float* nu, const float* r, const int32_t* active, float* out)
{
    if (p == nullptr || nu == nullptr || r == nullptr || out == nullptr || active == nullptr)
        return sil::fail(SIL_ERR_INVALID, "sil_precond_apply_active: NULL");
    std::vector<Sample> s;
    if (sil_status st = to_samples(samples, n, &s); st != SIL_OK) return st;
    return p->net.apply(s, nu, r, out, static_cast<cudaStream_t>(stream), active);
}

sil_status sil_precond_loss_grad(sil_precond p, sil_stream stream, const sil_precond_sample* samples, int n,
                                 const float* nu, const float* b, const float* x, double* loss,
                                 double* per_sample_loss, float* grad_host)
{
    if (p == nullptr || nu == nullptr || b == nullptr || x == nullptr || loss == nullptr)
        return sil::fail(SIL_ERR_INVALID, "sil_precond_loss_grad: NULL");
    std::vector<Sample> s;
    if (sil_status st = to_samples(samples, n, &s); st != SIL_OK) return st;
    std::vector<double> ps;
    cudaStream_t const cs = static_cast<cudaStream_t>(stream);
    sil_status st = p->net.loss_grad(s, nu, b, x, loss, &ps, cs);
    if (st != SIL_OK) return st;
    if (per_sample_loss != nullptr) std::copy(ps.begin(), ps.end(), per_sample_loss);
    if (grad_host != nullptr) {
        SIL_CUDA_CHECK(cudaMemcpyAsync(grad_host, p->net.grad, sizeof(float) * sil::nn::kNumParams,
                                       cudaMemcpyDeviceToHost, cs));
        SIL_CUDA_CHECK(cudaStreamSynchronize(cs));
    }
    return SIL_OK;
}

sil_status sil_precond_train_step(sil_precond p, sil_stream stream, const sil_precond_sample* samples, int n,
                                  const float* nu, const float* b, const float* x, float learning_rate, double* loss)
{
    if (p == nullptr || nu == nullptr || b == nullptr || x == nullptr || loss == nullptr || !(learning_rate > 0.0f))
        return sil::fail(SIL_ERR_INVALID, "sil_precond_train_step: bad argument");
    std::vector<Sample> s;
    if (sil_status st = to_samples(samples, n, &s); st != SIL_OK) return st;
    cudaStream_t const cs = static_cast<cudaStream_t>(stream);
    sil_status st = p->net.loss_grad(s, nu, b, x, loss, nullptr, cs);
    if (st != SIL_OK) return st;
    return p->net.adam_step(learning_rate, cs);
}

sil_status sil_precond_debug_fetch(sil_precond p, int which, int level, float* host, int64_t count)
{
    if (p == nullptr || host == nullptr) return sil::fail(SIL_ERR_INVALID, "sil_precond_debug_fetch: NULL");
    return p->net.debug_fetch(which, level, host, count, nullptr);
}

} // extern "C"
