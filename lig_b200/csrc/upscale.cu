// Gradient-aware Hermite-bicubic upscale (value, d/dx, d/dy, d2/dxdy planes,
// HWC with 3 channels, or 1 for the single-channel form of
// upscaler_torch.py:91-165), forward and backward.
//
// Coordinate maps:
//   mode 0  half-pixel over a ROI with the ROI extent truncated to int,
//           csrc/gradient_aware_upscaler.cu:201-218;
//   mode 1  align-corners (torch.linspace(0, n-1, steps)), upscaler_torch.py:108-122.
// Weights: C^-1 transposed times [1, t, t^2, t^3] (the Hermite basis),
// csrc/gradient_aware_upscaler.cu:137-154.
//
// Forward (48 B per source pixel + 12 B per output pixel): a thread owns one
// value (column, channel) of an output row and walks down up to 64 rows.  It
// reduces each source row along x once (8 values, read through L1; the next
// row's are on their way meanwhile) and keeps the two rows of the current
// cell in registers, so an output costs one shared weight vector, four
// products and one coalesced store, at any scale and without a staged window.
// x first, then y: the sum of csrc/gradient_aware_upscaler.cu:172-175 in
// another order.  2048^2 -> 8192^2: 796 us (8x64 tiles staged in shared
// memory, y first) -> 260; 2047x1535 -> 3070x2302: 221 -> 64.  Bound by
// instruction issue (75% of the slots) and the rows' load latency.
//
// Backward: a gather.  A thread owns one value of a texel row and walks the
// output rows that touch its CTA's texel rows: per row it reduces its column's
// cotangents along x (weights in registers, up to 8 columns loaded together),
// adds the two sums to the accumulators of the row's two texel rows, and
// writes a texel row once when the walk passes it.  No atomics, every texel
// written; the reference scatters 48 float atomics per output pixel
// (csrc/gradient_aware_upscaler.cu:313-370).  2047x1535 -> 3070x2302: 328 us
// (8x16 texels per CTA, patch staged in shared memory) -> 89; 512^2 -> 1024^2:
// 39 -> 12.  Bound by load latency (half the warps resident at 64 registers).
// Upscaling by more than four: upscale_bwd_wide_kernel.
#include <type_traits>

#include "common.cuh"

namespace lig {

__constant__ float kCinvF[16] = {1.f, 0.f, 0.f, 0.f, 0.f, 0.f, 1.f, 0.f,
                                 -3.f, 3.f, -2.f, -1.f, 2.f, -2.f, 1.f, 1.f};
__constant__ double kCinvD[16] = {1., 0., 0., 0., 0., 0., 1., 0.,
                                  -3., 3., -2., -1., 2., -2., 1., 1.};
template <typename T> __device__ __forceinline__ const T *cinv();
template <> __device__ __forceinline__ const float *cinv<float>() { return kCinvF; }
template <> __device__ __forceinline__ const double *cinv<double>() { return kCinvD; }

template <typename T>
__device__ __forceinline__ void hermite(T t, T (&w)[4]) {
    const T *C = cinv<T>();
    const T t2 = t * t;
    const T t3 = t2 * t;
    w[0] = C[0] * (T)1 + C[4] * t + C[8] * t2 + C[12] * t3;
    w[1] = C[1] * (T)1 + C[5] * t + C[9] * t2 + C[13] * t3;
    w[2] = C[2] * (T)1 + C[6] * t + C[10] * t2 + C[14] * t3;
    w[3] = C[3] * (T)1 + C[7] * t + C[11] * t2 + C[15] * t3;
}

struct UpMap {
    int mode, dst_n, src_n, roi_n;
    double lo;
    int flip = 0;  // backward: walk the output indices from the last one down
};

// Source coordinate of output index d (float arithmetic for T=float).
template <typename T>
__device__ __forceinline__ T src_coord(const UpMap &m, int d) {
    if (m.mode == 0) {
        return (T)m.lo + ((T)d + (T)0.5) * (T)m.roi_n / (T)m.dst_n - (T)0.5;
    }
    // torch.linspace(0, n-1, steps): two-sided evaluation, IEEE division
    if (m.dst_n == 1) return (T)0;
    T end = (T)(m.src_n - 1);
    T step;
    if (sizeof(T) == 4) step = (T)__fdiv_rn((float)end, (float)(m.dst_n - 1));
    else step = end / (T)(m.dst_n - 1);
    if (d < m.dst_n / 2) return step * (T)d;
    return end - step * (T)(m.dst_n - 1 - d);
}

template <typename T>
__device__ __forceinline__ void coord(const UpMap &m, int d, int &i0, int &i1, T (&w)[4]) {
    T s = src_coord<T>(m, d);
    int f = (int)Math<T>::floor_(s);
    T t = s - (T)f;
    i1 = max(0, min(f + 1, m.src_n - 1));
    i0 = max(0, min(f, m.src_n - 1));
    hermite<T>(t, w);
}

// ---------------------------------------------------------------- forward
constexpr int kUpThreads = 256;
constexpr int kFwdMaxRows = 64;  // 2048^2 -> 8192^2: 268 us with 64 rows a CTA, 292 with 32, 266 with 128
template <typename T> struct alignas(4 * sizeof(T)) W4 { T w[4]; };

template <typename T, int C, typename Off>
__global__ void __launch_bounds__(kUpThreads)
upscale_fwd_kernel(UpMap mx, UpMap my, int src_w, int rows, const T *__restrict__ f,
                   const T *__restrict__ fx, const T *__restrict__ fy,
                   const T *__restrict__ fxy, T *__restrict__ out) {
    __shared__ int2 s_y[kFwdMaxRows];
    __shared__ int s_end[kFwdMaxRows];
    __shared__ W4<T> s_cy[kFwdMaxRows];
    const int dst_w = mx.dst_n;
    const int r0 = blockIdx.y * rows, nrow = min(rows, my.dst_n - r0);
    if (threadIdx.x < nrow)
        coord<T>(my, r0 + threadIdx.x, s_y[threadIdx.x].x, s_y[threadIdx.x].y,
                 s_cy[threadIdx.x].w);
    const int64_t q = (int64_t)blockIdx.x * kUpThreads + threadIdx.x;
    const int c = (int)(q / C), ch = (int)(q - (int64_t)c * C);
    int x0, x1;
    T cx[4];
    coord<T>(mx, min(c, dst_w - 1), x0, x1, cx);
    __syncthreads();
    if (threadIdx.x < nrow) {  // the output rows of one source cell follow each other
        const int2 y = s_y[threadIdx.x];
        int e = threadIdx.x + 1;
        while (e < nrow && s_y[e].x == y.x && s_y[e].y == y.y) ++e;
        s_end[threadIdx.x] = e;
    }
    __syncthreads();
    if (c >= dst_w) return;
    // byte offsets in a plane: with 32 bits the four planes' loads share one
    // offset register (uniform base + offset), without 64-bit sums per load
    const Off pitch = (Off)src_w * (Off)(C * sizeof(T));
    const Off oa = (Off)(x0 * C + ch) * (Off)sizeof(T), ob = (Off)(x1 * C + ch) * (Off)sizeof(T);
    auto at = [](const T *p, Off o) {
        return *reinterpret_cast<const T *>(reinterpret_cast<const char *>(p) + o);
    };
    // the eight source values of row y at this output column, and from them
    // the row's value and y-derivative there
    auto fetch = [&](int y, T (&t)[8]) {
        const Off a = (Off)y * pitch + oa, b = (Off)y * pitch + ob;
        t[0] = at(f, a); t[1] = at(f, b); t[2] = at(fx, a); t[3] = at(fx, b);
        t[4] = at(fy, a); t[5] = at(fy, b); t[6] = at(fxy, a); t[7] = at(fxy, b);
    };
    auto reduce = [&](const T (&t)[8], T &v, T &d) {
        v = t[0] * cx[0] + t[1] * cx[1] + t[2] * cx[2] + t[3] * cx[3];
        d = t[4] * cx[0] + t[5] * cx[1] + t[6] * cx[2] + t[7] * cx[3];
    };
    int yb = -1;  // source row held in (vb, db)
    T va, da, vb = 0, db = 0;
    int yn = s_y[0].x;  // source row on its way in nx
    T nx[8];
    fetch(yn, nx);
    const int y_last = s_y[nrow - 1].y;
    auto at_row = [&](int y, T &v, T &d) {
        if (y != yn) fetch(y, nx);
        reduce(nx, v, d);
        yn = min(y + 1, y_last);
        fetch(yn, nx);
    };
    const int64_t o_pitch = (int64_t)dst_w * C;
    T *o = out + r0 * o_pitch + q;
    for (int r = 0; r < nrow;) {  // cell rows; s_y is the same for every thread
        const int2 y = s_y[r];
        if (y.x == yb) {
            va = vb;
            da = db;
        } else {
            at_row(y.x, va, da);
        }
        if (y.y == y.x) {
            vb = va;
            db = da;
        } else if (y.y != yb) {
            at_row(y.y, vb, db);
        }
        yb = y.y;
        const int end = s_end[r];
#pragma unroll 4
        for (; r < end; ++r, o += o_pitch) {
            const W4<T> cy = s_cy[r];
            *o = va * cy.w[0] + vb * cy.w[1] + da * cy.w[2] + db * cy.w[3];
        }
    }
}

// --------------------------------------------------------------- backward
constexpr int kBwdRowChunk = 32;  // output rows whose weights are staged at a time
constexpr int kBwdMaxRows = 32;   // texel rows a CTA walks (32 to 128 measured alike)

// A reversed ROI (roi_n < 0) maps output indices down the source; the backward
// (its FLIP instantiation) then numbers them from the last one, so that its maps
// always ascend.
template <bool FLIP> __device__ __forceinline__ int walk_index(const UpMap &m, int d) {
    return FLIP && m.flip ? m.dst_n - 1 - d : d;
}

template <typename T, bool FLIP>
__device__ __forceinline__ void coord_idx(const UpMap &m, int d, int &i0, int &i1) {
    T s = src_coord<T>(m, walk_index<FLIP>(m, d));
    int f = (int)Math<T>::floor_(s);
    i1 = max(0, min(f + 1, m.src_n - 1));
    i0 = max(0, min(f, m.src_n - 1));
}

// First output index in [0, dst_n] whose left (right: right) corner is >= s.
// The map ascends: from the inverse map's estimate a few steps find the
// index; a degenerate map, or an estimate further off, takes the binary search.
template <typename T, bool FLIP>
__device__ __forceinline__ int first_ge(const UpMap &m, int s, bool right) {
    auto ge = [&](int d) {
        int a, b;
        coord_idx<T, FLIP>(m, d, a, b);
        return (right ? b : a) >= s;
    };
    const int n = m.dst_n;
    const T x = (T)(right ? s - 1 : s);
    const T est = m.mode == 0 ? (x - (T)m.lo + (T)0.5) * (T)n / (T)m.roi_n - (T)0.5
                              : x * (T)(n - 1) / (T)max(m.src_n - 1, 1);
    if (m.mode != 0 || m.roi_n > 0) {
        int d = (int)max((T)0, min(est, (T)n));
        d = min(d, n);
#pragma unroll 1
        for (int k = 0; k < 4; ++k) {
            if (d < n && !ge(d)) ++d;
            else if (d > 0 && ge(d - 1)) --d;
            else return d;
        }
    }
    int lo = 0, hi = n;  // answer in [lo, hi]
#pragma unroll 1
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (ge(mid)) hi = mid; else lo = mid + 1;
    }
    return lo;
}

// Weights of output index d, with a clamped cell (both corners the same
// texel) folded into its first corner.
template <typename T, bool FLIP>
__device__ __forceinline__ void folded(const UpMap &m, int d, int &i0, int &i1, T (&w)[4]) {
    coord<T>(m, walk_index<FLIP>(m, d), i0, i1, w);
    if (i0 == i1) {
        w[0] += w[1];
        w[2] += w[3];
        w[1] = w[3] = (T)0;
    }
}

// One thread's walk over the output rows that touch its CTA's texel rows
// [sy0, sy1]: per row the x-reduction of its texel column (uv with the value
// weights, ud with the derivative weights, output columns ascending), added
// to the accumulators of the row's two texel rows; a texel row is written
// when the walk passes it.  NT > 0: the column has at most NT output columns,
// whose weights are kept in registers and whose values are loaded together,
// two rows at a time (a loop over a weight table that waits for every load
// took 140 us at 2047x1535 -> 3070x2302, against 89).
template <typename T>
struct BwdWalk {
    const T *g;          // this thread's first output column, first row of the walk
    int64_t g_pitch;     // to the walk's next row
    T *gf, *gfx, *gfy, *gfxy;
    int64_t o_pitch;     // values of a texel row
    bool active;
    int sy0, sy1, cur;   // texel rows of the CTA; acc0 belongs to row cur, acc1 to cur + 1
    T acc0[4], acc1[4];
    __device__ __forceinline__ void flush(int64_t q) {
        if (cur >= sy0 && cur <= sy1 && active) {
            const int64_t o = cur * o_pitch + q;
            gf[o] = acc0[0];
            gfx[o] = acc0[1];
            gfy[o] = acc0[2];
            gfxy[o] = acc0[3];
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            acc0[k] = acc1[k];
            acc1[k] = (T)0;
        }
        ++cur;
    }
    __device__ __forceinline__ void row(int64_t q, int2 y, const W4<T> &cy, T uv, T ud) {
        while (cur < y.x) flush(q);  // y is the same for every thread
        acc0[0] += uv * cy.w[0];
        acc0[1] += ud * cy.w[0];
        acc0[2] += uv * cy.w[2];
        acc0[3] += ud * cy.w[2];
        if (y.y != y.x) {
            acc1[0] += uv * cy.w[1];
            acc1[1] += ud * cy.w[1];
            acc1[2] += uv * cy.w[3];
            acc1[3] += ud * cy.w[3];
        }
    }
};

// FLIP: a reversed ROI, in x or y (mx.flip, my.flip)
template <typename T, int C, bool FLIP>
__global__ void __launch_bounds__(kUpThreads)
upscale_bwd_kernel(UpMap mx, UpMap my, int src_w, int src_h, int rows, const T *__restrict__ g,
                   T *__restrict__ gf, T *__restrict__ gfx, T *__restrict__ gfy,
                   T *__restrict__ gfxy) {
    __shared__ int s_rng[4];
    __shared__ int2 s_y[kBwdRowChunk];
    __shared__ W4<T> s_cy[kBwdRowChunk];
    const int tid = threadIdx.x, dst_w = mx.dst_n;
    const int64_t q = (int64_t)blockIdx.x * kUpThreads + tid;
    const int sy0 = blockIdx.y * rows, sy1 = min(sy0 + rows, src_h) - 1;
    if (tid == 0) s_rng[0] = first_ge<T, FLIP>(my, sy0, true);
    else if (tid == 32) s_rng[1] = first_ge<T, FLIP>(my, sy1 + 1, false) - 1;
    // this thread's texel column x: output columns [ia, im) have it as their
    // right corner, [im, ib) as their left one
    const int x = (int)min(q / C, (int64_t)src_w - 1), ch = (int)(q % C);
    const int ia = first_ge<T, FLIP>(mx, x, true), im = first_ge<T, FLIP>(mx, x, false),
              ib = first_ge<T, FLIP>(mx, x + 1, false);
    const int n = ib - ia;
    __syncthreads();
    const int j_lo = s_rng[0], j_hi = s_rng[1];
    const int CS = FLIP && mx.flip ? -C : C;  // to the walk's next column
    const int64_t pitch = (int64_t)dst_w * C;
    const T *g0 = g + (int64_t)walk_index<FLIP>(mx, ia) * C + ch +
                  (FLIP && my.flip ? (my.dst_n - 1) * pitch : 0);
    BwdWalk<T> B{g0, FLIP && my.flip ? -pitch : pitch, gf, gfx, gfy, gfxy, (int64_t)src_w * C,
                 q < (int64_t)src_w * C, sy0, sy1, sy0 - 1, {}, {}};
    auto weights = [&](int i, T &wv, T &wd) {  // of output column ia + i
        int x0, x1;
        T w[4];
        folded<T, FLIP>(mx, ia + i, x0, x1, w);
        wv = ia + i < im ? w[1] : w[0];
        wd = ia + i < im ? w[3] : w[2];
    };
    // FULL: every texel column of the CTA has exactly NT output columns
    auto walk = [&](auto nt_tag, auto full_tag) {
        constexpr int NT = decltype(nt_tag)::value;
        [[maybe_unused]] constexpr bool FULL = decltype(full_tag)::value;
        T wv[NT > 0 ? NT : 1], wd[NT > 0 ? NT : 1];
        if constexpr (NT > 0) {
#pragma unroll
            for (int k = 0; k < NT; ++k) {
                wv[k] = wd[k] = (T)0;
                if (k < n) weights(k, wv[k], wd[k]);
            }
        }
        for (int jb = j_lo; jb <= j_hi; jb += kBwdRowChunk) {
            const int nj = min(kBwdRowChunk, j_hi - jb + 1);
            __syncthreads();
            if (tid < nj) folded<T, FLIP>(my, jb + tid, s_y[tid].x, s_y[tid].y, s_cy[tid].w);
            __syncthreads();
            const T *gp = B.g + jb * B.g_pitch;
            if constexpr (NT > 0) {
                for (int j = 0; j < nj; j += 2, gp += 2 * B.g_pitch) {
                    const bool two = j + 1 < nj;
                    T v[2][NT];
#pragma unroll
                    for (int k = 0; k < NT; ++k) {
                        v[0][k] = FULL || k < n ? gp[k * CS] : (T)0;
                        v[1][k] = (FULL || k < n) && two ? gp[B.g_pitch + k * CS] : (T)0;
                    }
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        if (h == 1 && !two) break;
                        T uv = 0, ud = 0;
#pragma unroll
                        for (int k = 0; k < NT; ++k) {
                            uv += v[h][k] * wv[k];
                            ud += v[h][k] * wd[k];
                        }
                        B.row(q, s_y[j + h], s_cy[j + h], uv, ud);
                    }
                }
            } else {
                for (int j = 0; j < nj; ++j, gp += B.g_pitch) {
                    T uv = 0, ud = 0;
                    for (int i = 0; i < n; ++i) {
                        T a, b;
                        weights(i, a, b);
                        const T gv = gp[(int64_t)i * CS];
                        uv += gv * a;
                        ud += gv * b;
                    }
                    B.row(q, s_y[j], s_cy[j], uv, ud);
                }
            }
        }
        while (B.cur <= sy1) B.flush(q);
    };
    // the most output columns of a texel column in this CTA
    using std::false_type;
    using std::true_type;
    if (__syncthreads_and(n <= 4)) {
        if (__syncthreads_and(n == 4)) walk(std::integral_constant<int, 4>{}, true_type{});
        else walk(std::integral_constant<int, 4>{}, false_type{});
    } else if (__syncthreads_and(n <= 8)) {
        if (__syncthreads_and(n == 8)) walk(std::integral_constant<int, 8>{}, true_type{});
        else walk(std::integral_constant<int, 8>{}, false_type{});
    } else {
        walk(std::integral_constant<int, 0>{}, false_type{});
    }
}

// Strong upscaling, more than kBwdColumns output columns a texel: a warp takes a
// texel column.  Its lanes share the column's output values (contiguous in a
// row: ten columns of three channels, or 32 of one, at a time), K to a lane,
// with weights in registers; a lane sums its own share over the rows, and the
// lanes' sums meet when the walk leaves a texel row.  More than K columns a
// lane: further walks, which add to the texels.
// With one thread a value (upscale_bwd_kernel) every value of such a column
// recomputes its weights in each row, and small sources leave the chip idle.
// us with a patch staged per block of texels / one thread a value / this:
// 128^2 x 8 55 / 111 / 19, 512^2 x 8 488 / 221 / 165, 128^2 x 32 1190 / 2137 /
// 164, 64^2 x 64 5310 / 7700 / 230; a 64^2 crop of 1024^2 to 512^2 60 / 88 / 37.
// Up to kWideColumns columns and from kWideTexels texels on one thread a value
// stays ahead: 500^2 x 5 143 / 92 / 98, 1000^2 x 6.5 949 / 468 / 506 (400^2 x 5 97 /
// 64 / 63, 1000^2 x 7 1081 / 535 / 531).  Bound by issue (a row's sums, 20 of 30
// lanes at 8x) and the rows' loads.
constexpr int kWideWarps = 8, kBwdColumns = 8, kWideColumns = 13, kWideTexels = 200000;

template <int C, typename T> __device__ __forceinline__ T sum_slots(T t) {
    const unsigned FULL = 0xffffffffu;
    if constexpr (C == 1) {
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) t += __shfl_xor_sync(FULL, t, o);
        return t;
    } else {  // ten slots of three lanes; lanes 0..2 have the sums
        t += __shfl_down_sync(FULL, t, 15);
        const T fifth = __shfl_down_sync(FULL, t, 12);
        t += __shfl_down_sync(FULL, t, 6);
        t += __shfl_down_sync(FULL, t, 3);
        return t + fifth;
    }
}

template <typename T, int C, bool FLIP, int K>
__global__ void __launch_bounds__(32 * kWideWarps)
upscale_bwd_wide_kernel(UpMap mx, UpMap my, int src_w, int src_h, int rows,
                        const T *__restrict__ g, T *__restrict__ gf, T *__restrict__ gfx,
                        T *__restrict__ gfy, T *__restrict__ gfxy) {
    constexpr int SLOTS = 32 / C, U = K == 4 ? 2 : 4;  // U: rows loaded together
    static_assert(C == 1 || C == 3, "channels");
    __shared__ int2 s_y[kWideWarps][32];
    __shared__ W4<T> s_cy[kWideWarps][32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, dst_w = mx.dst_n;
    const int x = blockIdx.x * kWideWarps + w;
    const int sy0 = blockIdx.y * rows, sy1 = min(sy0 + rows, src_h) - 1;
    // lanes 0, 1: the texel rows' output rows [j_lo, j_hi); lanes 2..4: columns
    // [ia, im) have the texel as their right corner, [im, ib) as their left
    const int at = lane == 0 ? sy0 : lane == 1 ? sy1 + 1 : lane < 4 ? x : x + 1;
    const int found = first_ge<T, FLIP>(lane < 2 ? my : mx, at, lane == 0 || lane == 2);
    const unsigned ALL = 0xffffffffu;
    const int j_lo = __shfl_sync(ALL, found, 0), j_hi = __shfl_sync(ALL, found, 1);
    const int ia = __shfl_sync(ALL, found, 2), im = __shfl_sync(ALL, found, 3),
              ib = __shfl_sync(ALL, found, 4);
    const int64_t o_pitch = (int64_t)src_w * C;
    if (!__syncthreads_or(x < src_w && ia < ib && j_lo < j_hi)) {
        // the crop has no outputs near these texels
        const int first = blockIdx.x * kWideWarps, n = min(kWideWarps, src_w - first) * C;
        for (int i = threadIdx.x; i < n * (sy1 - sy0 + 1); i += blockDim.x) {
            const int64_t o = (sy0 + i / n) * o_pitch + first * C + i % n;
            gf[o] = gfx[o] = gfy[o] = gfxy[o] = (T)0;
        }
        return;
    }
    if (x >= src_w) return;  // (no CTA barriers below)
    const int slot = lane / C, ch = lane % C;
    const int64_t pitch = (int64_t)dst_w * C, down = FLIP && my.flip ? -pitch : pitch;
    const T *g0 = g + (FLIP && my.flip ? (my.dst_n - 1) * pitch : 0) + ch;
    const int64_t o_at = (int64_t)x * C + ch;
    int c0 = ia;
    do {
        T wv[K], wd[K];
        const T *gk[K];
        bool on[K];
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const int c = c0 + slot + k * SLOTS;
            on[k] = slot < SLOTS && c < ib;
            wv[k] = wd[k] = (T)0;
            gk[k] = g0 + (int64_t)walk_index<FLIP>(mx, on[k] ? c : ia) * C;
            if (on[k]) {
                int x0, x1;
                T cw[4];
                folded<T, FLIP>(mx, c, x0, x1, cw);
                wv[k] = c < im ? cw[1] : cw[0];
                wd[k] = c < im ? cw[3] : cw[2];
            }
        }
        T acc0[4] = {}, acc1[4] = {};
        int cur = sy0 - 1;  // acc0 belongs to texel row cur, acc1 to the next
        auto flush = [&]() {
            if (cur >= sy0 && cur <= sy1) {
                T t[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) t[k] = sum_slots<C>(acc0[k]);
                if (slot == 0) {
                    const int64_t o = cur * o_pitch + o_at;
                    const bool add = c0 > ia;
                    gf[o] = add ? gf[o] + t[0] : t[0];
                    gfx[o] = add ? gfx[o] + t[1] : t[1];
                    gfy[o] = add ? gfy[o] + t[2] : t[2];
                    gfxy[o] = add ? gfxy[o] + t[3] : t[3];
                }
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                acc0[k] = acc1[k];
                acc1[k] = (T)0;
            }
            ++cur;
        };
        for (int jb = j_lo; jb < j_hi; jb += 32) {
            const int nj = min(32, j_hi - jb);
            __syncwarp();
            if (lane < nj) folded<T, FLIP>(my, jb + lane, s_y[w][lane].x, s_y[w][lane].y, s_cy[w][lane].w);
            __syncwarp();
            for (int j = 0; j < nj; j += U) {
                T v[U][K];
#pragma unroll
                for (int u = 0; u < U; ++u)
#pragma unroll
                    for (int k = 0; k < K; ++k)
                        v[u][k] = on[k] && j + u < nj ? gk[k][(jb + j + u) * down] : (T)0;
#pragma unroll
                for (int u = 0; u < U; ++u) {
                    if (j + u >= nj) break;
                    const int2 y = s_y[w][j + u];
                    const W4<T> cy = s_cy[w][j + u];
                    T uv = 0, ud = 0;
#pragma unroll
                    for (int k = 0; k < K; ++k) {
                        uv += v[u][k] * wv[k];
                        ud += v[u][k] * wd[k];
                    }
                    while (cur < y.x) flush();  // y is the same for the whole warp
                    acc0[0] += uv * cy.w[0];
                    acc0[1] += ud * cy.w[0];
                    acc0[2] += uv * cy.w[2];
                    acc0[3] += ud * cy.w[2];
                    if (y.y != y.x) {
                        acc1[0] += uv * cy.w[1];
                        acc1[1] += ud * cy.w[1];
                        acc1[2] += uv * cy.w[3];
                        acc1[3] += ud * cy.w[3];
                    }
                }
            }
        }
        while (cur <= sy1) flush();
        c0 += SLOTS * K;
    } while (c0 < ib);
}

// Output columns of a texel away from the borders, at most.
inline int64_t columns_per_texel(const UpMap &m) {
    const int64_t out = m.mode == 0 ? m.dst_n : m.dst_n - 1;
    const int64_t src = m.mode == 0 ? (m.roi_n < 0 ? -(int64_t)m.roi_n : m.roi_n) : m.src_n - 1;
    return src > 0 ? (2 * out + src - 1) / src : m.dst_n;
}

template <typename T, int C, bool FLIP>
void upscale_bwd_wide(UpMap mx, UpMap my, int64_t columns, int src_h, int src_w, const T *g, T *gf,
                      T *gfx, T *gfy, T *gfxy, cudaStream_t s) {
    constexpr int SLOTS = 32 / C;
    int rows = 8;  // texel rows a warp walks: the most that leave 32 warps per SM
    while (rows > 1 && (int64_t)src_w * ((src_h + rows - 1) / rows) < 148 * 32) rows >>= 1;
    while ((src_h + rows - 1) / rows > 65535) rows <<= 1;  // (the grid's limit)
    const dim3 grid((src_w + kWideWarps - 1) / kWideWarps, (src_h + rows - 1) / rows);
    auto k = columns <= SLOTS       ? upscale_bwd_wide_kernel<T, C, FLIP, 1>
             : columns <= 2 * SLOTS ? upscale_bwd_wide_kernel<T, C, FLIP, 2>
                                   : upscale_bwd_wide_kernel<T, C, FLIP, 4>;
    k<<<grid, 32 * kWideWarps, 0, s>>>(mx, my, src_w, src_h, rows, g, gf, gfx, gfy, gfxy);
}

// Output (forward) or texel (backward) rows a CTA walks: the most, up to
// `most`, that leave at least 16 CTAs per SM.
inline int up_rows(int64_t row_values, int n_rows, int most) {
    const int64_t cols = (row_values + kUpThreads - 1) / kUpThreads;
    int r = most;
    while (r > 8 && cols * ((n_rows + r - 1) / r) < 148 * 16) r >>= 1;
    return r;
}

template <typename T, int C>
int upscale_fwd(int mode, int src_h, int src_w, int dst_h, int dst_w, double x1, double y1,
                double x2, double y2, const void *f, const void *fx, const void *fy,
                const void *fxy, void *out, cudaStream_t s) {
    // the reference truncates the ROI extent to int (csrc/gradient_aware_upscaler.cu:201-202)
    UpMap mx{mode, dst_w, src_w, (int)((T)x2 - (T)x1), (double)(T)x1};
    UpMap my{mode, dst_h, src_h, (int)((T)y2 - (T)y1), (double)(T)y1};
    const int64_t row = (int64_t)dst_w * C;
    const int rows = up_rows(row, dst_h, kFwdMaxRows);
    const dim3 grid((unsigned)((row + kUpThreads - 1) / kUpThreads), (dst_h + rows - 1) / rows);
    const bool small = (int64_t)src_h * src_w * C * (int64_t)sizeof(T) <= 0xffffffffll;
    auto k = small ? upscale_fwd_kernel<T, C, uint32_t> : upscale_fwd_kernel<T, C, uint64_t>;
    k<<<grid, kUpThreads, 0, s>>>(mx, my, src_w, rows, (const T *)f, (const T *)fx, (const T *)fy,
                                  (const T *)fxy, (T *)out);
    note_launches(1);
    LIG_LAUNCH_CHECK();
    return LIG_OK;
}

template <typename T, int C>
int upscale_bwd(int mode, int src_h, int src_w, int dst_h, int dst_w, double x1, double y1,
                double x2, double y2, const void *g, void *gf, void *gfx, void *gfy, void *gfxy,
                cudaStream_t s) {
    UpMap mx{mode, dst_w, src_w, (int)((T)x2 - (T)x1), (double)(T)x1};
    UpMap my{mode, dst_h, src_h, (int)((T)y2 - (T)y1), (double)(T)y1};
    mx.flip = mode == 0 && mx.roi_n < 0;
    my.flip = mode == 0 && my.roi_n < 0;
    const int64_t columns = columns_per_texel(mx);
    if (columns > kBwdColumns &&
        (columns > kWideColumns || (int64_t)src_h * src_w < kWideTexels)) {
        auto wide = mx.flip || my.flip ? upscale_bwd_wide<T, C, true> : upscale_bwd_wide<T, C, false>;
        wide(mx, my, columns, src_h, src_w, (const T *)g, (T *)gf, (T *)gfx, (T *)gfy, (T *)gfxy, s);
        note_launches(1);
        LIG_LAUNCH_CHECK();
        return LIG_OK;
    }
    const int64_t row = (int64_t)src_w * C;
    const int rows = up_rows(row, src_h, kBwdMaxRows);
    const dim3 grid((unsigned)((row + kUpThreads - 1) / kUpThreads), (src_h + rows - 1) / rows);
    auto k = mx.flip || my.flip ? upscale_bwd_kernel<T, C, true> : upscale_bwd_kernel<T, C, false>;
    k<<<grid, kUpThreads, 0, s>>>(mx, my, src_w, src_h, rows, (const T *)g, (T *)gf, (T *)gfx,
                                  (T *)gfy, (T *)gfxy);
    note_launches(1);
    LIG_LAUNCH_CHECK();
    return LIG_OK;
}

inline bool up_args_ok(int mode, int sh, int sw, int dh, int dw) {
    return (mode == 0 || mode == 1) && sh > 0 && sw > 0 && dh > 0 && dw > 0;
}

}  // namespace lig

using namespace lig;

namespace lig {
template <int C>
int upscale_fwd_dt(int dtype, int mode, int sh, int sw, int dh, int dw, double x1, double y1,
                   double x2, double y2, const void *f, const void *fx, const void *fy,
                   const void *fxy, void *out, cudaStream_t s) {
    if (dtype == LIG_F32)
        return upscale_fwd<float, C>(mode, sh, sw, dh, dw, x1, y1, x2, y2, f, fx, fy, fxy, out, s);
    if (dtype == LIG_F64)
        return upscale_fwd<double, C>(mode, sh, sw, dh, dw, x1, y1, x2, y2, f, fx, fy, fxy, out, s);
    return LIG_ERR_INVALID;
}
template <int C>
int upscale_bwd_dt(int dtype, int mode, int sh, int sw, int dh, int dw, double x1, double y1,
                   double x2, double y2, const void *g, void *gf, void *gfx, void *gfy,
                   void *gfxy, cudaStream_t s) {
    if (dtype == LIG_F32)
        return upscale_bwd<float, C>(mode, sh, sw, dh, dw, x1, y1, x2, y2, g, gf, gfx, gfy, gfxy, s);
    if (dtype == LIG_F64)
        return upscale_bwd<double, C>(mode, sh, sw, dh, dw, x1, y1, x2, y2, g, gf, gfx, gfy, gfxy,
                                      s);
    return LIG_ERR_INVALID;
}
}  // namespace lig

extern "C" int lig_upscale_fwd_nc(int dtype, int mode, int channels, int sh, int sw, int dh,
                                  int dw, double x1, double y1, double x2, double y2,
                                  const void *f, const void *fx, const void *fy, const void *fxy,
                                  void *out, void *stream) {
    if (!up_args_ok(mode, sh, sw, dh, dw) || !f || !fx || !fy || !fxy || !out) return LIG_ERR_INVALID;
    cudaStream_t s = (cudaStream_t)stream;
    if (channels == 3)
        return upscale_fwd_dt<3>(dtype, mode, sh, sw, dh, dw, x1, y1, x2, y2, f, fx, fy, fxy, out, s);
    if (channels == 1)
        return upscale_fwd_dt<1>(dtype, mode, sh, sw, dh, dw, x1, y1, x2, y2, f, fx, fy, fxy, out, s);
    return LIG_ERR_INVALID;
}

extern "C" int lig_upscale_bwd_nc(int dtype, int mode, int channels, int sh, int sw, int dh,
                                  int dw, double x1, double y1, double x2, double y2,
                                  const void *g, void *gf, void *gfx, void *gfy, void *gfxy,
                                  void *stream) {
    if (!up_args_ok(mode, sh, sw, dh, dw) || !g || !gf || !gfx || !gfy || !gfxy) return LIG_ERR_INVALID;
    cudaStream_t s = (cudaStream_t)stream;
    if (channels == 3)
        return upscale_bwd_dt<3>(dtype, mode, sh, sw, dh, dw, x1, y1, x2, y2, g, gf, gfx, gfy, gfxy, s);
    if (channels == 1)
        return upscale_bwd_dt<1>(dtype, mode, sh, sw, dh, dw, x1, y1, x2, y2, g, gf, gfx, gfy, gfxy, s);
    return LIG_ERR_INVALID;
}

extern "C" int lig_upscale_fwd(int dtype, int mode, int sh, int sw, int dh, int dw, double x1,
                               double y1, double x2, double y2, const void *f, const void *fx,
                               const void *fy, const void *fxy, void *out, void *stream) {
    return lig_upscale_fwd_nc(dtype, mode, 3, sh, sw, dh, dw, x1, y1, x2, y2, f, fx, fy, fxy, out,
                              stream);
}

extern "C" int lig_upscale_bwd(int dtype, int mode, int sh, int sw, int dh, int dw, double x1,
                               double y1, double x2, double y2, const void *g, void *gf,
                               void *gfx, void *gfy, void *gfxy, void *stream) {
    return lig_upscale_bwd_nc(dtype, mode, 3, sh, sw, dh, dw, x1, y1, x2, y2, g, gf, gfx, gfy,
                              gfxy, stream);
}
