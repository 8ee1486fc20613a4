// LIG level pipeline ops: the residual target between levels and the
// multi-level compose of a decode.
//
// Residual (train.py:113-126): resid = gt - up + 0.5, min-max normalised to
// [0, 1]; the level's store_min / store_max are the min and max.  Two passes
// over gt and up (the min/max reduction, then the normalised write) instead
// of six elementwise / reduction launches, vectorised (402 MB read at 4095x4093:
// 75 us; 603 MB read and written, some of it from L2: 84, 129 before); every value is computed with the
// same IEEE operations in the same order as the torch expression
// ((gt - up) + 0.5, then (r - lo) / (hi - lo) with a correctly rounded
// division), so the result is bit-identical.
//
// Compose (train.py:188-200): for level s > 0 the running image is resized
// to the level's size with bilinear half-pixel sampling (F.interpolate mode
// 'bilinear', align_corners=False: src = max((dst + 0.5) * in/out - 0.5, 0),
// right/bottom neighbour clamped) and the de-normalised level render
// clamp(render, 0, 1) * (hi - lo) - 0.5 + lo is added; the last level is
// clamped to [0, 1].  One pass per level, no intermediate resized image.
#include <cfloat>
#include <type_traits>

#include "common.cuh"

namespace lig {

constexpr int kLevelThreads = 256;
// Elementwise passes: 6 CTAs per SM, 4 vectors in flight per thread (4095x4093:
// minmax / normalise 75 / 84 us; 8 CTAs 75 / 87, 4 79 / 95, 2 in flight 74 / 99).
constexpr int kLevelCtas = 6, kLevelUnroll = 4;
// One value at a time (misaligned arrays): 16 CTAs from kScalarMany values on
// (normalise, 6 / 16: 1023^2 6.0 / 6.9 us, 2048^2 37 / 32, 4095^2 150 / 125).
constexpr int kScalarCtas = 16;
constexpr int64_t kScalarMany = 6000000;

__device__ __forceinline__ float atomic_min_f(float *a, float v) {
    // order-preserving int mapping of finite floats
    int *ai = reinterpret_cast<int *>(a);
    int old = *ai;
    while (__int_as_float(old) > v) {
        const int prev = atomicCAS(ai, old, __float_as_int(v));
        if (prev == old) break;
        old = prev;
    }
    return __int_as_float(old);
}

__device__ __forceinline__ float atomic_max_f(float *a, float v) {
    int *ai = reinterpret_cast<int *>(a);
    int old = *ai;
    while (__int_as_float(old) < v) {
        const int prev = atomicCAS(ai, old, __float_as_int(v));
        if (prev == old) break;
        old = prev;
    }
    return __int_as_float(old);
}

__global__ void minmax_init_kernel(float *mm) {
    mm[0] = FLT_MAX;
    mm[1] = -FLT_MAX;
}

// Elements are taken four at a time where the arrays are 16-byte aligned (VEC;
// the remainder, or everything otherwise, one at a time).
// pass 1: min / max of gt - up + 0.5 (NaNs are ignored by the comparisons)
template <bool VEC>
__global__ void __launch_bounds__(kLevelThreads)
resid_minmax_kernel(int64_t n, const float *__restrict__ gt, const float *__restrict__ up,
                    float *__restrict__ mm) {
    float lo = FLT_MAX, hi = -FLT_MAX;
    const int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t step = (int64_t)gridDim.x * blockDim.x;
    auto take = [&](float a, float b) {
        const float r = __fadd_rn(__fsub_rn(a, b), 0.5f);
        lo = fminf(lo, r);
        hi = fmaxf(hi, r);
    };
    const int64_t nv = VEC ? n / 4 : 0;
    const float4 *g4 = reinterpret_cast<const float4 *>(gt);
    const float4 *u4 = reinterpret_cast<const float4 *>(up);
#pragma unroll kLevelUnroll
    for (int64_t i = i0; i < nv; i += step) {
        const float4 a = g4[i], b = u4[i];
        take(a.x, b.x);
        take(a.y, b.y);
        take(a.z, b.z);
        take(a.w, b.w);
    }
    for (int64_t i = 4 * nv + i0; i < n; i += step) take(gt[i], up[i]);
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) {
        lo = fminf(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = fmaxf(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    __shared__ float s_lo[kLevelThreads / 32], s_hi[kLevelThreads / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) { s_lo[w] = lo; s_hi[w] = hi; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int k = 1; k < kLevelThreads / 32; ++k) { lo = fminf(lo, s_lo[k]); hi = fmaxf(hi, s_hi[k]); }
        lo = fminf(lo, s_lo[0]);
        hi = fmaxf(hi, s_hi[0]);
        atomic_min_f(mm, lo);
        atomic_max_f(mm + 1, hi);
    }
}

// pass 2: (r - lo) / (hi - lo), correctly rounded.  Walks from the end, where
// pass 1 stopped: up to the L2's size of the inputs is still there, and the
// streaming stores leave it there.
template <bool VEC>
__global__ void __launch_bounds__(kLevelThreads)
resid_normalise_kernel(int64_t n, const float *__restrict__ gt, const float *__restrict__ up,
                       const float *__restrict__ mm, float *__restrict__ out) {
    const float lo = mm[0], hi = mm[1];
    const float den = __fsub_rn(hi, lo);
    const int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t step = (int64_t)gridDim.x * blockDim.x;
    auto norm = [&](float a, float b) {
        const float r = __fadd_rn(__fsub_rn(a, b), 0.5f);
        return __fdiv_rn(__fsub_rn(r, lo), den);
    };
    const int64_t nv = VEC ? n / 4 : 0;
    const float4 *g4 = reinterpret_cast<const float4 *>(gt);
    const float4 *u4 = reinterpret_cast<const float4 *>(up);
    float4 *o4 = reinterpret_cast<float4 *>(out);
    for (int64_t i = 4 * nv + i0; i < n; i += step) out[i] = norm(gt[i], up[i]);
#pragma unroll kLevelUnroll
    for (int64_t i = nv - 1 - i0; i >= 0; i -= step) {
        const float4 a = g4[i], b = u4[i];
        __stcs(o4 + i, make_float4(norm(a.x, b.x), norm(a.y, b.y), norm(a.z, b.z),
                                   norm(a.w, b.w)));
    }
}

// Compose one level: out = base + (clamp(render) * (hi - lo) - 0.5 + lo),
// base = bilinear resize of prev [ph, pw, 3] to [H, W], prev itself when the
// sizes agree (compose_flat_kernel), or 0; clamp_out: final clamp to [0, 1].

// base + the de-normalised render of one value
struct ComposeOp {
    float lo, rng;
    int clamp_render, clamp_out;
    __device__ ComposeOp(const float *mm, float lo_h, float hi_h, int cr, int co)
        : lo(mm ? mm[0] : lo_h), clamp_render(cr), clamp_out(co) {
        rng = __fsub_rn(mm ? mm[1] : hi_h, lo);
    }
    __device__ float operator()(float base, float r) const {
        if (clamp_render) r = fminf(fmaxf(r, 0.f), 1.f);
        const float est = __fadd_rn(__fsub_rn(__fmul_rn(r, rng), 0.5f), lo);
        const float o = __fadd_rn(base, est);
        return clamp_out ? fminf(fmaxf(o, 0.f), 1.f) : o;
    }
};

// Without a resize (no previous level, or one of the same size) the rows do not
// matter: values in order, four at a time where the arrays are 16-byte aligned.
// 2048^2 with no previous level 14.6 us, against 18.5 with the row split below and
// 16.6 with one pixel a thread; 8192^2 261 with 16 CTAs per SM, 275 with 8, 280 with
// one pixel a thread.  Bound by HBM.
constexpr int kComposeFlatCtas = 16;
template <bool VEC>
__global__ void __launch_bounds__(kLevelThreads)
compose_flat_kernel(int64_t n, const float *__restrict__ prev, const float *__restrict__ render,
                    const float *__restrict__ mm, float lo_h, float hi_h, int clamp_render,
                    int clamp_out, float *__restrict__ out) {
    const ComposeOp op(mm, lo_h, hi_h, clamp_render, clamp_out);
    const int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int64_t step = (int64_t)gridDim.x * blockDim.x;
    const int64_t nv = VEC ? n / 4 : 0;
    const float4 *r4 = reinterpret_cast<const float4 *>(render);
    const float4 *p4 = reinterpret_cast<const float4 *>(prev);
    float4 *o4 = reinterpret_cast<float4 *>(out);
#pragma unroll kLevelUnroll
    for (int64_t i = i0; i < nv; i += step) {
        const float4 r = r4[i], b = prev ? p4[i] : make_float4(0.f, 0.f, 0.f, 0.f);
        o4[i] = make_float4(op(b.x, r.x), op(b.y, r.y), op(b.z, r.z), op(b.w, r.w));
    }
#pragma unroll kLevelUnroll
    for (int64_t i = 4 * nv + i0; i < n; i += step) out[i] = op(prev ? prev[i] : 0.f, render[i]);
}

// With a resize: a thread owns one value (column, channel) of a row — coalesced loads and
// stores — and walks kComposeRows rows, kComposeBatch of them with all their
// loads (the render's value and four taps of prev, which hit L1) on their way
// together.  The rows' taps and weights come from a table the CTA fills once:
// the float / integer conversions run at a quarter of the other operations'
// rate and cost more than the memory traffic when every value makes its own.
// Off: unsigned type of the byte offsets from a CTA's first row, and into prev.
// 4095x4093 from 2047x2046 (69 us of traffic): 92 us, against 115 with one
// pixel a thread and a 64-bit division each, 131 with the conversions per value
// and 146 with four flat values a thread.  Issue-bound (75% of the slots).
// Images of up to kNarrowValues values a row: a CTA is a whole row by as many
// groups of sixteen rows as it has threads for, so that few threads idle; the
// groups' rows alternate, so that a warp's loads lie side by side: 1000000x1 8.8 us
// and 100000x5 5.6 (8.4 and 5.5 with one pixel a thread, 82 and 15 with CTAs of 256
// columns).
constexpr int kComposeRows = 16, kComposeBatch = 4;  // 32 rows 95 us, batches of 2 / 8 98 / 104
constexpr int kNarrowValues = 128, kNarrowGroups = kLevelThreads / 3;
// Small images: groups of four rows where sixteen would leave fewer than two CTAs
// per SM (512^2 5.3 us instead of 6.2; 767x1023, four CTAs, 7.1 with sixteen and 8.3).
constexpr int kComposeFewRows = 4, kComposeFewCtas = 2;

template <typename Off> struct RowTap {
    Off a, b;        // byte offsets of the upper and lower row of prev
    float ly0, ly1;  // their weights
};

// NARROW: cw columns (a whole row) by kLevelThreads / cw groups, else one group.
template <typename Off, bool NARROW>
__global__ void __launch_bounds__(kLevelThreads)
compose_kernel(int rows, int cw, int ph, int pw, const float *__restrict__ prev, int H, int W,
               const float *__restrict__ render, const float *__restrict__ mm, float lo_h,
               float hi_h, int clamp_render, int clamp_out, float *__restrict__ out) {
    __shared__ RowTap<Off> s_row[kComposeRows * (NARROW ? kNarrowGroups : 1)];
    const int tid = threadIdx.x, groups = NARROW ? kLevelThreads / cw : 1;
    const int ty = NARROW ? tid / cw : 0, tx = NARROW ? tid - ty * cw : tid;
    const int64_t pitch = 3 * (int64_t)W;
    const Off q = NARROW ? (Off)tx : (Off)blockIdx.x * kLevelThreads + tx;
    // (the row blocks run over y and z of the grid: one dimension holds 65535)
    const int64_t rb = ((int64_t)blockIdx.z * gridDim.y + blockIdx.y) * (rows * groups);
    if (rb >= H) return;
    // the CTA's rows r0 .. r0 + n_rows - 1; group ty takes every groups-th
    const int r0 = (int)rb, n_rows = min(rows * groups, H - r0);
    const int nr = (n_rows - ty + groups - 1) / groups;
    // the half-pixel source index and weights written as the bilinear
    // definition states them (src = s (d + 0.5) - 0.5, negative -> 0;
    // lambda1 = src - floor, lambda0 = 1 - lambda1), so that the
    // compiler contracts them as it does torch's upsample kernel
    auto tap = [&](int k) {
        const float sh = __fdiv_rn((float)ph, (float)H);
        float ry = sh * ((float)(r0 + k) + 0.5f) - 0.5f;
        ry = ry < 0.f ? 0.f : ry;
        const int y0 = (int)ry, y1 = y0 + (y0 < ph - 1 ? 1 : 0);
        const float ly1 = ry - (float)y0;
        const Off p = (Off)pw * 12u;
        s_row[k] = RowTap<Off>{(Off)y0 * p, (Off)y1 * p, 1.f - ly1, ly1};
    };
    if (tid < n_rows) tap(tid);
    if constexpr (NARROW)
        for (int k = tid + kLevelThreads; k < n_rows; k += kLevelThreads) tap(k);
    const ComposeOp op(mm, lo_h, hi_h, clamp_render, clamp_out);
    const Off x = q / 3u, c = q - 3u * x;
    const float sw = __fdiv_rn((float)pw, (float)W);
    float rx = sw * ((float)x + 0.5f) - 0.5f;
    rx = rx < 0.f ? 0.f : rx;
    const int x0 = (int)rx;
    const float lx1 = rx - (float)x0, lx0 = 1.f - lx1;
    const Off oa = ((Off)3 * (Off)x0 + c) * 4u, ob = oa + (x0 < pw - 1 ? 12u : 0u);
    __syncthreads();
    if (NARROW ? ty >= groups : q >= pitch) return;
    auto at = [](const float *p, Off o) {
        return *reinterpret_cast<const float *>(reinterpret_cast<const char *>(p) + o);
    };
    // this CTA's rows: one base per array, offsets in bytes
    const float *rend = render + (r0 + ty) * pitch;
    float *dst = out + (r0 + ty) * pitch;
    const Off row = (Off)(pitch * 4 * groups);
    auto walk = [&](int k0, auto full_tag) {  // FULL: the whole batch lies inside
        constexpr bool FULL = decltype(full_tag)::value;
        float v[kComposeBatch], t[kComposeBatch][4];
#pragma unroll
        for (int k = 0; k < kComposeBatch; ++k) {
            if (!FULL && k0 + k >= nr) break;
            const Off o = (Off)(k0 + k) * row + (Off)q * 4u;
            v[k] = at(rend, o);
            const RowTap<Off> r = s_row[(k0 + k) * groups + ty];
            t[k][0] = at(prev, r.a + oa);
            t[k][1] = at(prev, r.a + ob);
            t[k][2] = at(prev, r.b + oa);
            t[k][3] = at(prev, r.b + ob);
        }
#pragma unroll
        for (int k = 0; k < kComposeBatch; ++k) {
            if (!FULL && k0 + k >= nr) break;
            const RowTap<Off> &rw = s_row[(k0 + k) * groups + ty];
            const float ly0 = rw.ly0, ly1 = rw.ly1;
            const float base =
                ly0 * (lx0 * t[k][0] + lx1 * t[k][1]) + ly1 * (lx0 * t[k][2] + lx1 * t[k][3]);
            *reinterpret_cast<float *>(reinterpret_cast<char *>(dst) + (Off)(k0 + k) * row +
                                       (Off)q * 4u) = op(base, v[k]);
        }
    };
    int k0 = 0;
    for (; k0 + kComposeBatch <= nr; k0 += kComposeBatch) walk(k0, std::true_type{});
    if (k0 < nr) walk(k0, std::false_type{});
}

inline int level_blocks(int64_t n, int ctas) {
    int64_t b = (n + kLevelThreads - 1) / kLevelThreads;
    const int64_t cap = 148 * ctas;
    return (int)(b < 1 ? 1 : (b > cap ? cap : b));
}

}  // namespace lig

using namespace lig;

extern "C" int lig_level_residual(int64_t n, const float *gt, const float *up, float *out,
                                  float *minmax, void *stream) {
    if (n <= 0 || !gt || !up || !out || !minmax) return LIG_ERR_INVALID;
    cudaStream_t s = (cudaStream_t)stream;
    minmax_init_kernel<<<1, 1, 0, s>>>(minmax);
    const bool vec = ((reinterpret_cast<uintptr_t>(gt) | reinterpret_cast<uintptr_t>(up) |
                       reinterpret_cast<uintptr_t>(out)) & 15) == 0;
    const int blocks = level_blocks(vec ? (n + 3) / 4 : n,
                                    vec || n < kScalarMany ? kLevelCtas : kScalarCtas);
    auto minmax_k = vec ? resid_minmax_kernel<true> : resid_minmax_kernel<false>;
    auto norm_k = vec ? resid_normalise_kernel<true> : resid_normalise_kernel<false>;
    minmax_k<<<blocks, kLevelThreads, 0, s>>>(n, gt, up, minmax);
    norm_k<<<blocks, kLevelThreads, 0, s>>>(n, gt, up, minmax, out);
    note_launches(3);
    LIG_LAUNCH_CHECK();
    return LIG_OK;
}

extern "C" int lig_level_compose(int prev_h, int prev_w, const float *prev, int H, int W,
                                 const float *render, const float *minmax, double store_min,
                                 double store_max, int clamp_render, int clamp_out, float *out,
                                 void *stream) {
    if (H <= 0 || W <= 0 || !render || !out || (prev && (prev_h <= 0 || prev_w <= 0)))
        return LIG_ERR_INVALID;
    cudaStream_t s = (cudaStream_t)stream;
    if (!prev || (prev_h == H && prev_w == W)) {
        const int64_t n = 3 * (int64_t)H * W;
        const bool vec = ((reinterpret_cast<uintptr_t>(prev) | reinterpret_cast<uintptr_t>(render) |
                           reinterpret_cast<uintptr_t>(out)) & 15) == 0;
        auto k = vec ? compose_flat_kernel<true> : compose_flat_kernel<false>;
        k<<<level_blocks(vec ? (n + 3) / 4 : n, kComposeFlatCtas), kLevelThreads, 0, s>>>(
            n, prev, render, minmax, (float)store_min, (float)store_max, clamp_render, clamp_out, out);
        note_launches(1);
        LIG_LAUNCH_CHECK();
        return LIG_OK;
    }
    const bool narrow = 3 * (int64_t)W <= kNarrowValues;
    const int cw = narrow ? 3 * W : kLevelThreads, groups = kLevelThreads / cw;
    const int64_t cols = narrow ? 1 : (3 * (int64_t)W + cw - 1) / cw;
    const int rows = cols * ((H + (int64_t)groups * kComposeRows - 1) / (groups * kComposeRows)) <
                             148 * kComposeFewCtas ? kComposeFewRows : kComposeRows;
    const int64_t row_blocks = ((int64_t)H + rows * groups - 1) / (rows * groups);
    const unsigned gz = (unsigned)((row_blocks + 65534) / 65535);
    const dim3 grid((unsigned)cols, (unsigned)((row_blocks + gz - 1) / gz), gz);
    // 32-bit byte offsets while a CTA's rows, and prev, lie within 4 GiB
    const bool small = 12 * (int64_t)W * kComposeRows <= 0xffffffffll &&
                       12 * (int64_t)prev_h * prev_w <= 0xffffffffll;
    auto k = small ? (narrow ? compose_kernel<uint32_t, true> : compose_kernel<uint32_t, false>)
                   : (narrow ? compose_kernel<uint64_t, true> : compose_kernel<uint64_t, false>);
    k<<<grid, kLevelThreads, 0, s>>>(rows, cw, prev_h, prev_w, prev, H, W, render, minmax,
                                     (float)store_min, (float)store_max, clamp_render, clamp_out,
                                     out);
    note_launches(1);
    LIG_LAUNCH_CHECK();
    return LIG_OK;
}
