// Weighted-sum rasterizer, forward and backward, plain and gradient-aware.
//
// Work decomposition (B200): one CTA per tile (or per work item of a
// batch's flattened (image, tile) list); the tile is split into <= 32
// regions of 32 lanes and warp w owns region w: 8x8 pixels with two pixels
// per lane in the sum forward (8x16 with four for many tiles) and, as a pair,
// in the gradient-aware forward; 8x4, 8x8 or 8x16 in the sum backward by tile
// count and density; the reference's warp in the gradient-aware backward,
// whose v_xy_abs is |sum over that warp| per Gaussian
// (csrc/gradient_aware_rasterizer.cu:317-341).
//
// Gaussian data: a pack kernel (or the projection of the fit step and of decode
// batches) writes one 16-byte-aligned 48-byte record per
// Gaussian (mean, conic, opacity, colour, cull half-widths, sigma
// threshold).  Forwards: each warp streams the tile's sorted id list in chunks
// of 32 records through shared memory, the next chunk in registers meanwhile.
// Backwards: the CTA stages batches of blockDim records.
//
// Culling: a warp runs only the Gaussians that can reach its region
// (forward: one ballot per 32 Gaussians, then the set bits in ascending, i.e.
// list, order; backward: a compacted per-warp list).  The test is a
// conservative box around the Gaussian's alpha >= 1/255 ellipse, built with
// margin (see finish_rec), refined by an exact ellipse-over-rectangle test, so every skipped pixel would have failed the
// reference's own `alpha < 1/255` test (csrc/forward.cu:258): results are
// unchanged.
//
// Per-pixel arithmetic follows the reference (csrc/forward.cu:250-269,
// csrc/backward.cu:102-150, csrc/gradient_aware_rasterizer.cu:201-315,
// :434-482), sigma with explicit roundings in its compiled form (sigma_ref),
// so that the alpha-threshold decisions are the same, and each pixel adds its
// terms in list order.
#include <mutex>
#include <tuple>
#include <type_traits>
#include <vector>

#include "adam.cuh"
#include "common.cuh"
#include "pair.cuh"
#include "project.cuh"

namespace lig {

// The fields every evaluation reads come first (two 16-byte loads); opacity
// and the cull data, read at staging or only with opacities, last.
template <typename T> struct alignas(16) Rec {
    T x, y, a, b;      // mean, conic (a, b)
    T c, r, g, bl;     // conic c, colour
    T o, wx, wy, thr;  // opacity, cull half-widths (negative: never cull), sigma threshold
};

// ------------------------------------------------------------ alpha cut
// The reference's per-pixel test rejects a term when sigma < 0 or
// min(clamp, __expf(-sigma)) < 1/255 (csrc/forward.cu:255-258,
// csrc/backward.cu:104-111); for clamp >= 1/255 the second half depends on
// __expf(-sigma) alone.  Over the non-negative floats that decision is a step
// in sigma's bit pattern: it passes below one pattern (the cut) and fails from
// it on, and every negative sigma (sign bit set) fails.  So for a sigma that
// is neither NaN nor -0, the whole test is one unsigned compare,
//   pass  <=>  bits(sigma) < cut.
// The cut is found on the device by the same expression: between 5.5
// (__expf(-5.5) = 0.00409, 4% above 1/255 — far beyond __expf's error) and 5.6
// (6% below) a warp narrows the bracket 32 ways per round (four rounds).
// lig_alpha_cut scans every non-negative float to show the decision is that
// step and that the search finds its edge (a GPU test).
__device__ __forceinline__ bool alpha_passes(float s) {
    return !(s < 0.f || fminf(0.999f, __expf(-s)) < 1.f / 255.f);
}

// One full warp; returns the cut (the first failing bit pattern) in every lane.
__device__ __forceinline__ uint32_t alpha_cut_search() {
    uint32_t lo = __float_as_uint(5.5f), hi = __float_as_uint(5.6f);  // pass(lo), fail(hi)
    const int lane = threadIdx.x & 31;
    while (hi - lo > 1) {
        const uint32_t step = (hi - lo + 31) / 32;
        const uint32_t cand = min(lo + (uint32_t)(lane + 1) * step, hi);
        const uint32_t fails = __ballot_sync(0xffffffffu, !alpha_passes(__uint_as_float(cand)));
        const int f = __ffs(fails) - 1;  // hi itself fails, so some lane does
        const uint32_t new_hi = __shfl_sync(0xffffffffu, cand, f);
        if (f > 0) lo = __shfl_sync(0xffffffffu, cand, f - 1);
        hi = new_hi;
    }
    return hi;
}

// The cut on this device, written by every float pack launch (always the same
// value) and read by the rasterizer launched after it on the same stream.
__device__ uint32_t g_alpha_cut;

// The fused fit step's optimiser scalars (out null: not wanted).
// skipped_host: pinned host copy of *skipped.
struct AdamPro {
    const int32_t *status;
    int32_t *steps, *skipped, *skipped_host;
    double lr, b1, b2;
    AdamScalars *out = nullptr;
};

__device__ __forceinline__ void fit_prologue(const AdamPro &pro, int n_img) {
    adam_prologue(threadIdx.x, n_img, pro.status, pro.steps, pro.skipped, pro.lr, pro.b1, pro.b2,
                  pro.out);
    if (threadIdx.x == 0) *pro.skipped_host = *pro.skipped;
}

// ------------------------------------------------------------------ pack
// Culling data: the alpha >= 1/255 region of a positive-definite conic is the
// ellipse sigma <= t/2, t = 2 ln(255 o), whose x half-extent is sqrt(t Sxx).
// With t_c = max(t, 0.01) the record carries the box half-widths
// w = 1.001 sqrt(t_c Sxx) + 2 px and the sigma threshold
// thr = 1.001 t_c/2 + 0.02: a pixel with sigma > thr has
// alpha < exp(-0.02)/255, i.e. 2% below the reference's 1/255 cut, far beyond
// the rounding of sigma and __expf, so skipping it changes nothing.  No culling (w < 0) for non-finite inputs, non-positive
// opacity, non-positive-definite or nearly degenerate conics (b^2 > 0.999 ac),
// where the reference's per-pixel tests must run everywhere in the tile, nor
// where a conic entry times the squared reach of the box (plus a 16-pixel
// region) could approach the float range.  A record with culling data
// (w >= 0) therefore has a finite positive-definite conic and finite sigma
// terms, so at every pixel it is evaluated on, sigma is finite and not -0
// (every term of sigma_ref / sigma_half is >= +0 except b dx dy, and their
// sum is +0 or a positive normal or negative float): the alpha cut's compare
// applies.
// HALF: the record carries a/2 and c/2 in place of a and c (the fused-loss
// forward, see sigma_half); the cull data are computed from the full conic.
// zero (backward): also clears the Gaussian's zero_stride accumulators there
// (zero_stride * sizeof(T) a multiple of 16 bytes, 16-byte aligned).
// ticket (fused loss): cleared for the loss kernel.
// Float: block 0's first warp also publishes the alpha cut.
// TAME (the packed gradient-aware kernels, which add a zero where a pixel
// fails the alpha test instead of skipping it): culling data only for records
// whose products at any pixel they are evaluated on stay finite (see
// kTameSlope, kTameColor), so that the zero weight yields a zero; the others
// take the kernels' skipping walk.
constexpr float kTameSlope = 1e6f;  // largest conic entry times the reach: |sx|, |sy| < 2e6
constexpr float kTameColor = 1e8f;
constexpr float kTameCot = 1e12f;  // larger (or non-finite) cotangents: the skipping walks

template <typename T>
__device__ __forceinline__ bool tame_cotangent(T a, T b, T c, T d) {
    return fabs(a) < (T)kTameCot && fabs(b) < (T)kTameCot && fabs(c) < (T)kTameCot &&
           fabs(d) < (T)kTameCot;
}

__device__ __forceinline__ void publish_alpha_cut() {  // first warp of the grid
    if (blockIdx.x == 0 && threadIdx.x < 32) {
        const uint32_t cut = alpha_cut_search();
        if (threadIdx.x == 0) g_alpha_cut = cut;
    }
}

// Completes a record whose inputs are set: the culling data, and with HALF the
// halved conic.
template <typename T, bool HALF, bool TAME>
__device__ __forceinline__ void finish_rec(Rec<T> &r) {
    r.thr = 0;
    double a = r.a, b = r.b, c = r.c, o = r.o;
    double det = a * c - b * b;
    bool ok = isfinite((double)r.x) && isfinite((double)r.y) && isfinite(a) && isfinite(b) &&
              isfinite(c) && isfinite(o) && o > 0.0 && a > 0.0 && c > 0.0 && det > 0.0 &&
              b * b <= 0.999 * a * c && fabs(r.x) < 1e7 && fabs(r.y) < 1e7;
    T wx = (T)-1, wy = (T)-1;
    if (ok) {
        double t = 2.0 * log(255.0 * o);
        double tc = t > 0.01 ? t : 0.01;
        double sxx = c / det, syy = a / det;
        double hx = 1.001 * sqrt(tc * sxx) + 2.0, hy = 1.001 * sqrt(tc * syy) + 2.0;
        const float reach = (float)fmax(hx, hy) + 16.f;
        const float entry = fmaxf(fmaxf((float)r.a, (float)r.c), fabsf((float)r.b));
        const bool tame = !TAME || (entry * reach < kTameSlope && (float)fabs(r.r) < kTameColor &&
                                    (float)fabs(r.g) < kTameColor && (float)fabs(r.bl) < kTameColor);
        if (hx < 1e7 && hy < 1e7 && entry * reach * reach < 1e36f && tame) {
            wx = (T)hx;
            wy = (T)hy;
            r.thr = (T)(0.5 * tc * 1.001 + 0.02);
        }
    }
    r.wx = wx;
    r.wy = wy;
    if (HALF) {
        r.a *= (T)0.5;
        r.c *= (T)0.5;
    }
}


template <typename T, bool HALF, bool TAME = false>
__global__ void pack_kernel(int n, const T *__restrict__ xys, const T *__restrict__ conics,
                            const T *__restrict__ colors, const T *__restrict__ opac,
                            Rec<T> *__restrict__ recs, T *__restrict__ zero, int zero_stride,
                            uint32_t *__restrict__ ticket) {
    if (ticket && blockIdx.x == 0 && threadIdx.x == 32) *ticket = 0;
    if (sizeof(T) == 4) publish_alpha_cut();
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (zero) {
        float4 *z = reinterpret_cast<float4 *>(zero + (size_t)i * zero_stride);
        const int nv = zero_stride * (int)sizeof(T) / 16;
        for (int k = 0; k < nv; ++k) z[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    Rec<T> r;
    r.x = xys[2 * i];
    r.y = xys[2 * i + 1];
    r.a = conics[3 * i];
    r.b = conics[3 * i + 1];
    r.c = conics[3 * i + 2];
    r.o = opac ? opac[i] : (T)1;
    r.r = colors[3 * i];
    r.g = colors[3 * i + 1];
    r.bl = colors[3 * i + 2];
    finish_rec<T, HALF, TAME>(r);
    recs[i] = r;
}

// Projection (as project_fwd_kernel's) and the forward's record of Gaussian k of
// a set, number i of the batch, in image im.  A Gaussian outside its image
// leaves a zero count only: nothing reads its other outputs, except those of
// each image's first, which phantom slots name (slot_id in binning.cu).
template <bool VIEW>
__device__ __forceinline__ void project_rec(const BatchGeo &geo, int im, int i, int k, bool chol,
                                            const float *in3, const float *means, float o,
                                            const float *rgb, const View<float> &view,
                                            float *__restrict__ xys, float *__restrict__ extents,
                                            int32_t *__restrict__ counts,
                                            Rec<float> *__restrict__ recs) {
    float cx, cy, cz;
    input_cov<float, VIEW>(chol, in3, k, cx, cy, cz, view);
    float mx = means[2 * k], my = means[2 * k + 1];
    if constexpr (VIEW) {
        mx = (mx - view.ox) * view.sx;
        my = (my - view.oy) * view.sy;
    }
    Rec<float> r;
    float ex = 0, ey = 0;
    r.a = r.b = r.c = 0;
    const bool ok = cov2d_bounds(cx, cy, cz, o, r.a, r.b, r.c, ex, ey);
    int32_t area = 0;
    if (ok) {
        int x0, y0, x1, y1;
        tile_bbox(mx, my, ex, ey, (unsigned)geo.tbx[im], (unsigned)geo.tby(im), (unsigned)geo.B, x0,
                  y0, x1, y1);
        area = (int32_t)((unsigned)(x1 - x0) * (unsigned)(y1 - y0));
    } else {
        r.a = r.b = r.c = 0;
    }
    const bool hit = area > 0;
    counts[i] = hit ? area : 0;
    if (!hit && i != geo.g_off[im]) return;
    r.x = hit ? mx : 0.f;
    r.y = hit ? my : 0.f;
    xys[2 * i] = r.x;
    xys[2 * i + 1] = r.y;
    extents[2 * i] = hit ? ex : 0.f;
    extents[2 * i + 1] = hit ? ey : 0.f;
    r.o = o;
    r.r = rgb[3 * k];
    r.g = rgb[3 * k + 1];
    r.bl = rgb[3 * k + 2];
    finish_rec<float, true, false>(r);
    recs[i] = r;
}

// The views of a batch of decodes, each with its own set and transform, in one
// launch, one CTA per 256 Gaussians of one view.
// Bound by the records' fp64 and the reads of every Gaussian.  Eight views of
// 500k Gaussians: 71 us, against 44 for eight projections, 51 for the colours'
// copies and 54 for packing every record.
struct ViewSet {
    const float *in3, *means, *opac, *rgb;
    float ox, oy, sx, sy;
    int chol;
};
struct ViewSets {
    int block_off[kMaxBatch + 1];
    ViewSet v[kMaxBatch];
};

__global__ void __launch_bounds__(256)
project_views_kernel(const BatchGeo geo, const ViewSets sets, float *__restrict__ xys,
                     float *__restrict__ extents, int32_t *__restrict__ counts,
                     Rec<float> *__restrict__ recs) {
    publish_alpha_cut();
    const int im = BatchGeo::find(sets.block_off, geo.n_img, blockIdx.x);
    const int k = (blockIdx.x - sets.block_off[im]) * blockDim.x + threadIdx.x;
    const int i = geo.g_off[im] + k;
    if (i >= geo.g_off[im + 1]) return;
    const ViewSet &s = sets.v[im];
    const View<float> view{s.ox, s.oy, s.sx, s.sy, true};
    project_rec<true>(geo, im, i, k, s.chol != 0, s.in3, s.means, s.opac ? s.opac[k] : 1.f, s.rgb,
                      view, xys, extents, counts, recs);
}

// The fit step's first kernel: projection and records, the backward's gradient
// sums cleared, and the words that the scan, the binning and the loss launch
// start from.
// HBM-bound.  8192^2 / 2M: 51 us (132 B a Gaussian: 40), against 18 + 37 for
// projection and packing; 512^2 / 50k: the step 104 -> 96 us, three launches fewer.
__global__ void __launch_bounds__(256)
fit_project_kernel(const BatchGeo geo, int n, const float *__restrict__ params,
                   float *__restrict__ xys, float *__restrict__ extents,
                   int32_t *__restrict__ counts, Rec<float> *__restrict__ recs,
                   float4 *__restrict__ sums, uint32_t *__restrict__ scan_state, int n_state,
                   int32_t *__restrict__ status, uint32_t *__restrict__ ticket) {
    publish_alpha_cut();
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n_state) scan_state[i] = 0;
    if (i == 0) {
        *status = 0;
        *ticket = 0;
    }
    if (i >= n) return;
    sums[2 * (size_t)i] = sums[2 * (size_t)i + 1] = make_float4(0.f, 0.f, 0.f, 0.f);
    project_rec<false>(geo, geo.image_of_gauss(i), i, i, true, params + 2 * (size_t)n, params, 1.f,
                       params + 5 * (size_t)n, View<float>{0, 0, 1, 1, false}, xys, extents,
                       counts, recs);
}

// ---------------------------------------------------------------- regions
// A tile is split into R <= 32 regions of 32 pixels; warp w of the CTA owns
// region w and each lane owns PPL pixels of it.
//   kind 0: 8x4 blocks, PPL 1               (backward; gradient-aware forward)
//   kind 1: 8x8 blocks, lane owns (x, y) and (x, y + 4)  (sum forward)
//   kind 3: 8x16 blocks, lane owns (x, y + 4p), p < 4   (sum forward, large images)
//   kind 2: the reference's warps, thread ranks 32w..32w+31 with
//           rank = ty*B + tx, PPL 1                    (gradient-aware backward)
struct Regions {
    int kind, B, nbx, nby, count;
    __host__ __device__ static Regions make(int kind, int B) {
        Regions r{kind, B, 1, 1, 1};
        if (kind == 0) { r.nbx = (B + 7) / 8; r.nby = (B + 3) / 4; }
        else if (kind == 1) { r.nbx = (B + 7) / 8; r.nby = (B + 7) / 8; }
        else if (kind == 3) { r.nbx = (B + 7) / 8; r.nby = (B + 15) / 16; }
        else { r.nbx = 1; r.nby = (B * B + 31) / 32; }
        r.count = r.nbx * r.nby;
        return r;
    }
    __device__ __forceinline__ void pixel(int w, int lane, int p, int &lx, int &ly) const {
        if (kind == 0) {
            lx = (w % nbx) * 8 + (lane & 7);
            ly = (w / nbx) * 4 + (lane >> 3);
        } else if (kind == 1 || kind == 3) {
            lx = (w % nbx) * 8 + (lane & 7);
            ly = (w / nbx) * block_h() + (lane >> 3) + 4 * p;
        } else {
            int r = w * 32 + lane;
            lx = r % B;
            ly = r < B * B ? r / B : B;  // B marks "no pixel"
        }
    }
    // rows of a block region (kinds 0, 1, 3)
    __host__ __device__ __forceinline__ int block_h() const {
        return kind == 0 ? 4 : (kind == 1 ? 8 : 16);
    }
    // tile-local pixel-centre rectangle of region w (conservative)
    template <typename T>
    __device__ __forceinline__ void rect(int w, T &x0, T &x1, T &y0, T &y1) const {
        int ix0, ix1, iy0, iy1;
        if (kind == 2) {
            const int r0 = w * 32, r1 = min(w * 32 + 31, B * B - 1);
            iy0 = r0 / B; iy1 = r1 / B;
            if (iy0 == iy1) { ix0 = r0 % B; ix1 = r1 % B; }
            else { ix0 = 0; ix1 = B - 1; }
        } else {
            const int hb = block_h();
            ix0 = (w % nbx) * 8; ix1 = min(ix0 + 7, B - 1);
            iy0 = (w / nbx) * hb; iy1 = min(iy0 + hb - 1, B - 1);
        }
        x0 = (T)ix0 + (T)0.5; x1 = (T)ix1 + (T)0.5;
        y0 = (T)iy0 + (T)0.5; y1 = (T)iy1 + (T)0.5;
    }
    __device__ __forceinline__ uint32_t all() const {
        return count >= 32 ? 0xffffffffu : ((1u << count) - 1u);
    }
    // Regions whose pixel centres (tile-local, pixel i at i + 0.5) can lie in
    // the box [x0, x1] x [y0, y1].  Conservative.
    template <typename T>
    __device__ __forceinline__ uint32_t bits(T x0, T x1, T y0, T y1) const {
        if (kind == 2) {
            // rows j with centre in [y0, y1]; a region spans rows r0/B .. r1/B
            T fy0 = Math<T>::ceil_(y0 - (T)0.5), fy1 = Math<T>::floor_(y1 - (T)0.5);
            if (!(fy0 <= fy1) || fy1 < (T)0 || fy0 > (T)(B - 1)) return 0u;
            int j0 = (int)max(fy0, (T)0), j1 = (int)min(fy1, (T)(B - 1));
            uint32_t m = 0;
            for (int w = 0; w < count; ++w) {
                int r0 = (w * 32) / B, r1 = min(w * 32 + 31, B * B - 1) / B;
                if (r0 <= j1 && r1 >= j0) m |= 1u << w;
            }
            return m;
        }
        const int hb = block_h();
        T c0 = Math<T>::ceil_((x0 - (T)7.5) / (T)8), c1 = Math<T>::floor_((x1 - (T)0.5) / (T)8);
        T r0 = Math<T>::ceil_((y0 - ((T)hb - (T)0.5)) / (T)hb);
        T r1 = Math<T>::floor_((y1 - (T)0.5) / (T)hb);
        c0 = max(c0, (T)0); r0 = max(r0, (T)0);
        c1 = min(c1, (T)(nbx - 1)); r1 = min(r1, (T)(nby - 1));
        if (!(c0 <= c1) || !(r0 <= r1)) return 0u;
        int ic0 = (int)c0, ic1 = (int)c1, ir0 = (int)r0, ir1 = (int)r1;
        uint32_t cols = ((1u << (ic1 - ic0 + 1)) - 1u) << ic0;
        uint32_t m = 0;
        for (int r = ir0; r <= ir1; ++r) m |= cols << (r * nbx);
        return m;
    }
};

// Minimum of sigma(d) = 0.5 (a dx^2 + c dy^2) + b dx dy over the rectangle
// [dx0, dx1] x [dy0, dy1] (positive-definite conic): zero if the rectangle
// holds the origin, else the least of the edge minima (each a clamped 1-D
// quadratic minimum).
// With the centre outside the rectangle the minimum lies on an edge that
// faces the centre (at the minimiser every active bound's inward move must
// not decrease sigma, while the direction to the centre does; that direction
// points outward only across facing edges), so at most one vertical and one
// horizontal edge are evaluated: x = dx0 when dx0 > 0, x = dx1 when dx1 < 0,
// and likewise in y.
template <typename T>
__device__ __forceinline__ T sigma_min_rect(T a, T b, T c, T dx0, T dx1, T dy0, T dy1) {
    const bool ox = dx0 > (T)0 || dx1 < (T)0, oy = dy0 > (T)0 || dy1 < (T)0;
    if (!ox && !oy) return (T)0;
    T best = (T)3.0e38;
    if (ox) {
        const T dx = dx0 > (T)0 ? dx0 : dx1;
        const T dy = min(max(-b * dx / c, dy0), dy1);
        best = (T)0.5 * (a * dx * dx + c * dy * dy) + b * dx * dy;
    }
    if (oy) {
        const T dy = dy0 > (T)0 ? dy0 : dy1;
        const T dx = min(max(-b * dy / a, dx0), dx1);
        best = min(best, (T)0.5 * (a * dx * dx + c * dy * dy) + b * dx * dy);
    }
    return best;
}

// Region mask of one Gaussian for the tile at pixel origin (tx0, ty0): the
// regions whose pixel-centre rectangle meets the Gaussian's cull box and, on
// it, reaches sigma <= thr (see finish_rec: every pixel with sigma > thr
// fails the reference's own alpha >= 1/255 test).  Records without culling
// data (wx < 0) touch every region.
// ELLIPSE = false stops at the box test.  HALF: the record carries the
// halved conic (fused-loss forward).
template <typename T, bool ELLIPSE = true, bool HALF = false>
__device__ __forceinline__ uint32_t region_bits(const Rec<T> &g, const Regions &R, int tx0,
                                                int ty0) {
    if (!(g.wx >= (T)0)) return R.all();
    const T cx = g.x - (T)tx0, cy = g.y - (T)ty0;
    uint32_t m = R.bits<T>(cx - g.wx, cx + g.wx, cy - g.wy, cy + g.wy);
    if (!ELLIPSE) return m;
    uint32_t keep = m;
    while (m) {
        const int w = __ffs(m) - 1;
        m &= m - 1;
        T x0, x1, y0, y1;
        R.rect<T>(w, x0, x1, y0, y1);
        const T a = HALF ? (T)2 * g.a : g.a, c = HALF ? (T)2 * g.c : g.c;
        if (sigma_min_rect<T>(a, g.b, c, x0 - cx, x1 - cx, y0 - cy, y1 - cy) > g.thr)
            keep &= ~(1u << w);
    }
    return keep;
}

// One region's test of region_bits: does the Gaussian reach region w?
template <typename T, bool ELLIPSE, bool HALF>
__device__ __forceinline__ bool region_hit(const Rec<T> &g, const Regions &R, int w, int tx0,
                                           int ty0) {
    if (!(g.wx >= (T)0)) return true;
    T x0, x1, y0, y1;
    R.rect<T>(w, x0, x1, y0, y1);
    const T cx = g.x - (T)tx0, cy = g.y - (T)ty0;
    if (cx + g.wx < x0 || cx - g.wx > x1 || cy + g.wy < y0 || cy - g.wy > y1) return false;
    if (!ELLIPSE) return true;
    const T a = HALF ? (T)2 * g.a : g.a, c = HALF ? (T)2 * g.c : g.c;
    return !(sigma_min_rect<T>(a, g.b, c, x0 - cx, x1 - cx, y0 - cy, y1 - cy) > g.thr);
}

// ------------------------------------------------------------ tile setup
// Work item -> image and tile origin.  Work items index the flattened
// (image, tile) list of a BatchGeo; a single image is a batch of one.
struct TileCtx {
    int im, H, W, B, tx0, ty0, poff;
    bool empty;  // the image has no intersections (reference empty-list branch)
};

// Intersections of image im: from the inclusive prefix sum of per-Gaussian
// counts when given (batched), else the whole list's total.
__device__ __forceinline__ bool image_empty(const BatchGeo &geo, const int32_t *cum,
                                            const int32_t *d_total, int im) {
    if (!cum) return *d_total == 0;
    const int g0 = geo.g_off[im], g1 = geo.g_off[im + 1];
    if (g1 <= g0) return true;
    const int hi = cum[g1 - 1], lo = g0 > 0 ? cum[g0 - 1] : 0;
    return hi - lo == 0;
}

__device__ __forceinline__ TileCtx tile_ctx(const BatchGeo &geo, const int32_t *cum,
                                            const int32_t *d_total, int tile) {
    TileCtx t;
    t.im = geo.image_of_tile(tile);
    const int lt = tile - geo.tile_off[t.im];
    const int tbx = geo.tbx[t.im];
    t.H = geo.H[t.im];
    t.W = geo.W[t.im];
    t.B = geo.B;
    t.tx0 = (lt % tbx) * t.B;
    t.ty0 = (lt / tbx) * t.B;
    t.poff = geo.pix_off[t.im];
    t.empty = image_empty(geo, cum, d_total, t.im);
    return t;
}

// Next work item: blockIdx.x in a plain launch (one CTA per tile); in a
// persistent launch (work != null) the CTA pulls items from a global counter
// until the list is exhausted.  The loop ends because the counter only grows.
__device__ __forceinline__ int next_tile(int *work, int &s_slot, bool first) {
    if (!work) return first ? (int)blockIdx.x : 0x7fffffff;
    __syncthreads();  // everyone is done with the previous item
    if (threadIdx.x == 0) s_slot = atomicAdd(work, 1);
    __syncthreads();
    return s_slot;
}

// --------------------------------------------------------------- forward
#ifndef LIG_RASTER_FWD_ELLIPSE
#define LIG_RASTER_FWD_ELLIPSE 1  // sum forward: exact ellipse test per region
#endif
#ifndef LIG_RASTER_FWD_ELLIPSE_GA
#define LIG_RASTER_FWD_ELLIPSE_GA 1  // the same in the gradient-aware forward
#endif
#ifndef LIG_RASTER_ALPHA_CUT
#define LIG_RASTER_ALPHA_CUT 1  // forwards without opacities: alpha test by the cut's compare
#endif
// One CTA per tile, warp w = region w (8x4 pixels), one pixel per lane.
// Batches of blockDim Gaussians (list order) are staged in shared memory, one
// record per thread, with the next batch's record fetched into registers
// while the current batch is processed.  Each thread also stores its
// Gaussian's region mask; a warp then walks only the Gaussians whose mask has
// its bit (ballot over the batch, set bits in ascending order = list order),
// two per iteration so the two sigma/alpha chains overlap, accumulating in
// list order — per pixel exactly the reference's sequence of additions.
// sigma = 0.5 (a dx^2 + c dy^2) + b dx dy (csrc/forward.cu:250-251,
// csrc/backward.cu:102-104, csrc/gradient_aware_rasterizer.cu:201-203),
// rounded step by step as the reference's expression compiles under
// --use_fast_math: fma(b dx, dy, 0.5 fma(a dx, dx, (c dy) dy)) — established by
// comparing the compiled expression against each explicit form on 4M random
// inputs.  Written explicitly so that the surrounding code (several pixels
// per lane sharing products) cannot change the contraction, and with it the
// alpha >= 1/255 decisions.
// Rounded product / fused multiply-add, spelled out so that the compiler
// cannot contract or reassociate them.
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) {
    return __fma_rn(a, b, c);
}

template <typename T>
__device__ __forceinline__ T sigma_ref(T a, T b, T c, T dx, T dy);
template <>
__device__ __forceinline__ float sigma_ref<float>(float a, float b, float c, float dx, float dy) {
    const float ta = __fmul_rn(a, dx), tc = __fmul_rn(c, dy), tb = __fmul_rn(b, dx);
    return __fmaf_rn(tb, dy, __fmul_rn(0.5f, __fmaf_rn(ta, dx, __fmul_rn(tc, dy))));
}
template <>
__device__ __forceinline__ double sigma_ref<double>(double a, double b, double c, double dx,
                                                    double dy) {
    const double ta = __dmul_rn(a, dx), tc = __dmul_rn(c, dy), tb = __dmul_rn(b, dx);
    return __fma_rn(tb, dy, __dmul_rn(0.5, __fma_rn(ta, dx, __dmul_rn(tc, dy))));
}

// sigma_ref from the halved conic (ha = a/2, hc = c/2):
//   fma(b dx, dy, fma(ha dx, dx, (hc dy) dy)) == fma(b dx, dy, 0.5 fma(a dx, dx, (c dy) dy))
// bit for bit — halving is exact and commutes with rounding (away from the
// subnormal range, where every term is far below any alpha decision) — with
// one product fewer.
template <typename T>
__device__ __forceinline__ T sigma_half(T ha, T b, T hc, T dx, T dy) {
    return fma_rn(mul_rn(b, dx), dy, fma_rn(mul_rn(ha, dx), dx, mul_rn(mul_rn(hc, dy), dy)));
}

template <typename T>
struct PixelEval {
    // gradient-aware, csrc/gradient_aware_rasterizer.cu:436-445 (d = p - mu);
    // returns false when the term is skipped.
    static __device__ __forceinline__ bool alpha(const Rec<T> &g, T px, T py, T &dx, T &dy,
                                                 T &a) {
        using M = Math<T>;
        dx = px - g.x;
        dy = py - g.y;
        const T sigma = sigma_ref<T>(g.a, g.b, g.c, dx, dy);
        a = M::min_((T)0.999, g.o * M::exp_(-sigma));
        return !(sigma < (T)0 || a < (T)1 / (T)255);
    }
};

template <typename T, bool GA>
struct FwdAcc {
    T r = 0, g = 0, b = 0, w = 0;
    T dx[GA ? 3 : 1] = {}, dy[GA ? 3 : 1] = {}, dxy[GA ? 3 : 1] = {};
    int cur = 0;
    // sum: colour, with FIN the final index and with WS the weight sum
    template <bool FIN, bool WS>
    __device__ __forceinline__ void add_sum(const Rec<T> &q, T a, int idx) {
        // csrc/forward.cu:264-269
        r += q.r * a;
        g += q.g * a;
        b += q.bl * a;
        if constexpr (WS) w += a;
        if constexpr (FIN) cur = idx;
    }
    __device__ __forceinline__ void add(const Rec<T> &q, T dxp, T dyp, T a, int idx) {
        // csrc/gradient_aware_rasterizer.cu:451-482
        r += q.r * a;
        g += q.g * a;
        b += q.bl * a;
        if (GA) {
            const T sdx = q.a * dxp + q.b * dyp;
            const T sdy = q.b * dxp + q.c * dyp;
            const T s2 = q.b;
            const T adx = -a * sdx;
            const T ady = -a * sdy;
            const T adxy = -a * (s2 - sdx * sdy);
            dx[0] += q.r * adx; dx[1] += q.g * adx; dx[2] += q.bl * adx;
            dy[0] += q.r * ady; dy[1] += q.g * ady; dy[2] += q.bl * ady;
            dxy[0] += q.r * adxy; dxy[1] += q.g * adxy; dxy[2] += q.bl * adxy;
        }
        w += a;
        cur = idx;
    }
};

// Fused clamped-L2 loss in the forward (fit loops): instead of the image the
// forward writes the masked difference diff = (0 <= x <= 1) ? clamp(x) - t : 0
// (what the loss gradient needs per pixel) and each tile adds
// (clamp(x) - t)^2 over its pixels into one fp64 partial (fixed-order block
// reduction, so the loss is deterministic).  No target: plain forward.
// An 8-bit target (an RGB image as stored) is read as t = byte / 255 rounded
// to nearest: the float value torchvision's ToTensor gives (train.py's image
// loading), so the result equals the fp32 path fed that float target.  In
// float the quotient is q = b * r (r = 1/255 rounded) refined by one
// residual-correction step (Markstein): e = fma(-q, 255, b), t = fma(e, r, q)
// — equal to the correctly rounded b / 255 for every byte b (checked against
// the host's division for all 256 values), with no division.
// A batch of decodes: each view's image is its own allocation.
struct ViewImages {
    float *img[kMaxBatch];
};

template <typename T> struct L2Fwd {
    const T *target;
    double *tile_partial;  // [total tiles]
    const uint8_t *target_u8 = nullptr;
    __device__ __forceinline__ bool on() const { return target || target_u8; }
    __device__ __forceinline__ T at(int i) const;
};
template <> __device__ __forceinline__ float L2Fwd<float>::at(int i) const {
    if (!target_u8) return target[i];
    constexpr float r = 0.003921568859368563f;  // 1/255 rounded to nearest (0x3b808081)
    const float b = (float)target_u8[i];
    const float q = __fmul_rn(b, r);
    return __fmaf_rn(__fmaf_rn(-q, 255.0f, b), r, q);
}
template <> __device__ __forceinline__ double L2Fwd<double>::at(int i) const {
    return target_u8 ? __ddiv_rn((double)target_u8[i], 255.0) : target[i];
}

template <typename T>
__device__ __forceinline__ void block_sum_to(double v, double *dst) {
    __shared__ double s_part[32];
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) s_part[w] = v;
    __syncthreads();
    if (threadIdx.x == 0) {
        double t = 0;
        for (int k = 0; k < (int)(blockDim.x >> 5); ++k) t += s_part[k];
        *dst = t;
    }
    __syncthreads();
}

// Writes one pixel's forward outputs, or in the fused-L2 mode its masked
// difference; returns the pixel's (clamp(x) - t)^2 sum for the tile partial.
template <typename T, bool GA>
__device__ __forceinline__ double fwd_write(const FwdAcc<T, GA> &acc, bool inside, int pix,
                                            T *__restrict__ img, T *__restrict__ wsum,
                                            T *__restrict__ odx, T *__restrict__ ody,
                                            T *__restrict__ odxy,
                                            int32_t *__restrict__ final_idx,
                                            const L2Fwd<T> &l2) {
    if (!inside) return 0.0;
    if (final_idx) final_idx[pix] = acc.cur;
    if (l2.on()) {
        double sq = 0;
        const T x[3] = {acc.r, acc.g, acc.b};
#pragma unroll
        for (int ch = 0; ch < 3; ++ch) {
            const T d = min(max(x[ch], (T)0), (T)1) - l2.at(3 * pix + ch);
            sq += (double)(d * d);
            img[3 * pix + ch] = (x[ch] >= (T)0 && x[ch] <= (T)1) ? d : (T)0;
        }
        return sq;
    }
    img[3 * pix] = acc.r;
    img[3 * pix + 1] = acc.g;
    img[3 * pix + 2] = acc.b;
    if (wsum) wsum[pix] = acc.w;
    if (GA) {
#pragma unroll
        for (int ch = 0; ch < 3; ++ch) {
            odx[3 * pix + ch] = acc.dx[ch];
            ody[3 * pix + ch] = acc.dy[ch];
            odxy[3 * pix + ch] = acc.dxy[ch];
        }
    }
    return 0.0;
}

// PPL pixels per lane: 1 (8x4 regions, two Gaussians per iteration; gradient-
// aware), 2 (8x8 regions, lane owns (x, y) and (x, y + 4)) or 4 (8x16, (x, y +
// 4p)); each Gaussian's record and loop overhead are shared by the lane's
// evaluations, whose independent sigma / exp chains overlap.  Per pixel the
// terms are added in list order either way.
// The sum forward's records carry the halved conic (see sigma_half); a lane's
// pixels share their column, so dx, (a/2) dx and b dx are formed once per
// Gaussian.  OP: opacities.  FIN, WS: final indices and weight sums are wanted
// (the fused loss needs neither).  Without opacities, chunks whose records all
// carry culling data test alpha by the cut's compare: bound by instruction
// issue; eight views of 500k Gaussians with weight sums and indices 401 us, against
// 498 with the full conic, an opacity product and the float test.
template <typename T, bool GA, int PPL, bool OP, bool FIN, bool WS>
__device__ __forceinline__ void fwd_tile(const TileCtx &tc, int tile, const int32_t *__restrict__ ids,
                                         const int2 *__restrict__ tile_bins,
                                         const Rec<T> *__restrict__ recs, T *__restrict__ img,
                                         T *__restrict__ wsum, T *__restrict__ odx,
                                         T *__restrict__ ody, T *__restrict__ odxy,
                                         int32_t *__restrict__ final_idx, Rec<T> *s_rec,
                                         const L2Fwd<T> &l2, uint32_t cut) {
    constexpr bool kCut = !GA && !OP && sizeof(T) == 4 && LIG_RASTER_ALPHA_CUT;
    const unsigned FULL = 0xffffffffu;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const int B = tc.B, tx0 = tc.tx0, ty0 = tc.ty0;
    static_assert(GA ? PPL == 1 : PPL == 2 || PPL == 4, "pixels per lane");
    const Regions R = Regions::make(PPL == 1 ? 0 : (PPL == 2 ? 1 : 3), B);
    // a warp lists only the Gaussians whose alpha >= 1/255 ellipse meets
    // its region (one test per Gaussian and region)
    constexpr bool ELL = LIG_RASTER_FWD_ELLIPSE && (!GA || LIG_RASTER_FWD_ELLIPSE_GA);
    bool inside[PPL];
    int pix[PPL];
    T px[PPL], py[PPL];
#pragma unroll
    for (int p = 0; p < PPL; ++p) {
        int lx, ly;
        R.pixel(w, lane, p, lx, ly);
        const int gx = tx0 + lx, gy = ty0 + ly;
        inside[p] = lx < B && ly < B && gx < tc.W && gy < tc.H;
        pix[p] = tc.poff + gy * tc.W + gx;
        px[p] = (T)gx + (T)0.5;
        py[p] = (T)gy + (T)0.5;
    }

    FwdAcc<T, GA> acc[PPL];
    // walk the Gaussians of `mask` (bits of the 32 records at rb, list
    // indices ib + bit) in list order; fast_tag true: every record has
    // culling data, so alpha is tested by the cut's compare
    auto walk = [&](uint32_t mask, const Rec<T> *rb, int ib, auto fast_tag) {
        [[maybe_unused]] constexpr bool FAST = decltype(fast_tag)::value;
        if constexpr (!GA) {
            using M = Math<T>;
            while (mask) {
                const int b1 = __ffs(mask) - 1;
                mask &= mask - 1;
                const Rec<T> g1 = rb[b1];
                const T dx = g1.x - px[0];
                const T hadx = mul_rn(g1.a, dx), bdx = mul_rn(g1.b, dx);
                T ap[PPL];
                bool okp[PPL];
#pragma unroll
                for (int p = 0; p < PPL; ++p) {
                    const T dy = g1.y - py[p];
                    const T sg = fma_rn(bdx, dy, fma_rn(hadx, dx, mul_rn(mul_rn(g1.c, dy), dy)));
                    const T e = M::exp_(-sg);
                    ap[p] = M::min_((T)0.999, OP ? g1.o * e : e);
                    if constexpr (FAST) okp[p] = __float_as_uint((float)sg) < cut;
                    else okp[p] = !(sg < (T)0 || ap[p] < (T)1 / (T)255);
                }
#pragma unroll
                for (int p = 0; p < PPL; ++p)
                    if (okp[p]) acc[p].template add_sum<FIN, WS>(g1, ap[p], ib + b1);
            }
        } else {
            while (mask) {
                const int b1 = __ffs(mask) - 1;
                mask &= mask - 1;
                const Rec<T> g1 = rb[b1];
                T dx1, dy1, a1;
                const bool ok1 = PixelEval<T>::alpha(g1, px[0], py[0], dx1, dy1, a1);
                if (mask) {
                    const int b2 = __ffs(mask) - 1;
                    mask &= mask - 1;
                    const Rec<T> g2 = rb[b2];
                    T dx2, dy2, a2;
                    const bool ok2 = PixelEval<T>::alpha(g2, px[0], py[0], dx2, dy2, a2);
                    if (ok1) acc[0].add(g1, dx1, dy1, a1, ib + b1);
                    if (ok2) acc[0].add(g2, dx2, dy2, a2, ib + b2);
                } else if (ok1) {
                    acc[0].add(g1, dx1, dy1, a1, ib + b1);
                }
            }
        }
    };
    if (!tc.empty) {
        const int2 range = tile_bins[tile];
        // each warp streams the tile's list in chunks of 32 on its own
        // (its region's test only, no block barriers: warps whose
        // regions have short lists do not wait for the others)
        Rec<T> *w_rec = s_rec + w * 32;
        Rec<T> pre;
        if (range.x + lane < range.y) pre = recs[__ldg(ids + range.x + lane)];
        for (int base = range.x; base < range.y; base += 32) {
            const bool hit =
                base + lane < range.y && region_hit<T, ELL, !GA>(pre, R, w, tx0, ty0);
            // a chunk whose records all carry culling data takes the cut
            bool fast = false;
            if constexpr (kCut)
                fast = !__any_sync(FULL, base + lane < range.y && !(pre.wx >= (T)0));
            __syncwarp();
            w_rec[lane] = pre;
            __syncwarp();
            if (base + 32 + lane < range.y) pre = recs[__ldg(ids + base + 32 + lane)];
            const uint32_t mask = __ballot_sync(FULL, hit);
            if (kCut && fast) walk(mask, w_rec, base, std::bool_constant<kCut>{});
            else walk(mask, w_rec, base, std::false_type{});
        }
    } else {  // the reference's empty-list branch (rasterize.py:80-90)
#pragma unroll
        for (int p = 0; p < PPL; ++p) acc[p].r = acc[p].g = acc[p].b = (T)1;
    }
    double sq = 0.0;
#pragma unroll
    for (int p = 0; p < PPL; ++p)
        sq += fwd_write<T, GA>(acc[p], inside[p], pix[p], img, wsum, odx, ody, odxy, final_idx, l2);
    if (l2.on()) block_sum_to<T>(sq, l2.tile_partial + tile);
}

// Launch bounds: tiles of B <= 16 launch <= 256 threads, and their
// instantiations ask for a number of resident CTAs per SM (the register budget
// follows); larger tiles use instantiations for more threads.
#ifndef LIG_RASTER_FWD_MINB
#define LIG_RASTER_FWD_MINB 4
#endif
#ifndef LIG_RASTER_BWD_LEAN_MINB
#define LIG_RASTER_BWD_LEAN_MINB 4  // the paired loop wants the larger register budget
#endif
// From LIG_RASTER_BWD_LARGE_MIN_TILES tiles on, the lean backward asks for
// LIG_RASTER_BWD_LEAN_MINB_LARGE resident CTAs per SM (fewer registers, a few
// spilled, more warps to hide latency): measured 4% faster at 8192^2 and
// 1% at 2048^2, but 14% slower at 512^2 (1024 tiles).
#ifndef LIG_RASTER_BWD_LEAN_MINB_LARGE
#define LIG_RASTER_BWD_LEAN_MINB_LARGE 5  // pairs + bulk-staged records (48 registers)
#endif
#ifndef LIG_RASTER_BWD_LARGE_MIN_TILES
#define LIG_RASTER_BWD_LARGE_MIN_TILES 4096
#endif
#ifndef LIG_RASTER_BWD_RROWS
#define LIG_RASTER_BWD_RROWS 0  // float lean walks of large images: region rows (4, 8, 16; 0: by density)
#endif
// Region rows by density (Gaussians per pixel): taller regions save per-pair
// work, but evaluate more pixels a pair cannot reach, which costs more when
// the tile lists are long.  Whole calls on 16x16 tiles with 8x16 / 8x8 regions, us:
// lean walk at 0.03 Gaussians per pixel (8192^2, 2M) 1940 / 2092, at 0.04 (4096^2)
// 643 / 613, 0.06 937 / 818, 0.24 (2048^2, 1M) 896 / 722; general walk 2551 / 3013,
// 816 / 922, 1225 / 1169, 1163 / 940.  The crossover is near 0.036 for the lean walks
// and 0.046 for the general one; the line lies between.
#ifndef LIG_RASTER_BWD_R16_MAX_DENSITY
#define LIG_RASTER_BWD_R16_MAX_DENSITY 0.04
#endif
#ifndef LIG_RASTER_BWD_RROWS_MINB
// resident CTAs per SM of the 8x8 walk (128 threads): 2048^2 / 1M 681 us with 7
// (72 registers), 696 with 6, 705 with 8 (64, spilling)
#define LIG_RASTER_BWD_RROWS_MINB 7
#endif
#ifndef LIG_RASTER_BWD_R16_MINB
#define LIG_RASTER_BWD_R16_MINB 14  // resident CTAs per SM of the 8x16 walk (64 threads, 72 registers)
#endif
// Resident CTAs per SM of the general walk (opacities, wsum cotangent), 8x4 /
// 8x8 / 8x16 regions.  767x1023 / 150k: 4 CTAs 103 us, 3 107, 2 120 (150 for
// the scalar walk); 2048^2 / 500k (8x8): 6 540, 7 532, 5 518 (726); 2048^2 /
// 100k (8x16): 12 148, 14 147, 10 149 (243).
#ifndef LIG_RASTER_GEN_MINB
#define LIG_RASTER_GEN_MINB 4
#endif
#ifndef LIG_RASTER_GEN_R8_MINB
#define LIG_RASTER_GEN_R8_MINB 5
#endif
#ifndef LIG_RASTER_GEN_R16_MINB
#define LIG_RASTER_GEN_R16_MINB 12
#endif
#ifndef LIG_RASTER_BWD_SPLIT2
#define LIG_RASTER_BWD_SPLIT2 8  // with up to this many Gaussians left, 4 lanes take one
#endif
#ifndef LIG_RASTER_BWD_R16_SPLIT1
#define LIG_RASTER_BWD_R16_SPLIT1 32  // the 8x16 walk: 2 lanes per Gaussian at least
#endif
#ifndef LIG_RASTER_BWD_R16_SPLIT3
#define LIG_RASTER_BWD_R16_SPLIT3 8  // the 8x16 walk: 8 lanes per Gaussian from this many left
#endif
#ifndef LIG_RASTER_BWD_SPLIT3
#define LIG_RASTER_BWD_SPLIT3 4  // with up to this many Gaussians left, 8 lanes take one
#endif
#ifndef LIG_RASTER_BWD_SPLIT
#define LIG_RASTER_BWD_SPLIT 1  // split a short list's Gaussians across lanes (measured faster)
#endif
#ifndef LIG_RASTER_BWD_SPLIT1
#define LIG_RASTER_BWD_SPLIT1 24  // with up to this many Gaussians left, 2 lanes take one
#endif
#ifndef LIG_RASTER_BWD_LANE_ELLIPSE
#define LIG_RASTER_BWD_LANE_ELLIPSE 1  // ellipse culling by the warp's lanes (measured faster)
#endif
#ifndef LIG_RASTER_BWD_MINB
#define LIG_RASTER_BWD_MINB 5
#endif

// Sum forward: two pixels per lane, four from LIG_RASTER_PPL4_MIN_TILES tiles on
// (fewer warps per tile, so small images keep more pixels in flight with fewer
// pixels per lane).
#ifndef LIG_RASTER_PPL4_MIN_TILES
#define LIG_RASTER_PPL4_MIN_TILES 4096  // measured: faster from 2048^2 up, not at 512^2
#endif

// Resident CTAs per SM asked of the register allocator.  Forward (128 threads),
// 2048^2 / 1M and 512^2 / 50k: 8 CTAs (64 registers) 973 / 41 us, 9 968 / 43,
// 7 990 / 40, 6 1110 / 47, 10 1110 / 49.  Backward (256 threads), 2047x1535 /
// 190k and 512^2 / 50k with opacities: 3 CTAs 518 / 67 us, 2 552 / 64.
#ifndef LIG_RASTER_GA_MINB
#define LIG_RASTER_GA_MINB 8
#endif
#ifndef LIG_RASTER_GA_BWD_MINB
#define LIG_RASTER_GA_BWD_MINB 3
#endif
// Lanes per Gaussian as in the lean walk; two lanes from 32 left on measured
// 586 against 552 us, 20 / 12 / 6 left 558 (2047x1535).
#ifndef LIG_RASTER_GA_BWD_SPLIT1
#define LIG_RASTER_GA_BWD_SPLIT1 24
#endif
#ifndef LIG_RASTER_GA_BWD_SPLIT2
#define LIG_RASTER_GA_BWD_SPLIT2 8
#endif
#ifndef LIG_RASTER_GA_BWD_SPLIT3
#define LIG_RASTER_GA_BWD_SPLIT3 4
#endif

template <typename T, bool GA, int PPL, int MAXT, int MINB, bool OP = true, bool FIN = true,
          bool WS = true>
__global__ void __launch_bounds__(MAXT, MINB)
raster_fwd_kernel(const BatchGeo geo, const int32_t *__restrict__ cum, int *work,
                  const int32_t *__restrict__ ids, const int2 *__restrict__ tile_bins,
                  const int32_t *__restrict__ d_total, const Rec<T> *__restrict__ recs,
                  T *__restrict__ img, T *__restrict__ wsum, T *__restrict__ odx,
                  T *__restrict__ ody, T *__restrict__ odxy, int32_t *__restrict__ final_idx,
                  L2Fwd<T> l2) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int s_slot;
    Rec<T> *s_rec = reinterpret_cast<Rec<T> *>(smem_raw);
    const int n_tiles = geo.total_tiles();
    const uint32_t cut = !GA && !OP && sizeof(T) == 4 ? g_alpha_cut : 0u;
    for (int tile = next_tile(work, s_slot, true); tile < n_tiles;
         tile = next_tile(work, s_slot, false)) {
        const TileCtx tc = tile_ctx(geo, cum, d_total, tile);
        fwd_tile<T, GA, PPL, OP, FIN, WS>(tc, tile, ids, tile_bins, recs, img, wsum, odx, ody,
                                          odxy, final_idx, s_rec, l2, cut);
    }
}

// The sum forward of a batch of decodes, images only (no weight sums, no final
// indices), each into its own allocation: eight views of 500k Gaussians 355 us,
// against 401 with both, and no copies out of a shared buffer (55 us).
template <int PPL, int MAXT, int MINB, bool OP>
__global__ void __launch_bounds__(MAXT, MINB)
raster_views_kernel(const BatchGeo geo, const int32_t *__restrict__ cum,
                    const int32_t *__restrict__ ids, const int2 *__restrict__ tile_bins,
                    const Rec<float> *__restrict__ recs, const ViewImages out) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    TileCtx tc = tile_ctx(geo, cum, nullptr, blockIdx.x);
    tc.poff = 0;
    fwd_tile<float, false, PPL, OP, false, false>(
        tc, blockIdx.x, ids, tile_bins, recs, out.img[tc.im], nullptr, nullptr, nullptr, nullptr,
        nullptr, reinterpret_cast<Rec<float> *>(smem_raw), L2Fwd<float>{nullptr, nullptr},
        OP ? 0u : g_alpha_cut);
}

// Gradient-aware forward, float: 8x8 regions, the lane's two pixels (x, y) and
// (x, y + 4) evaluated as a pair with f32x2 operations.  Per pixel the alphas,
// their order and the colour sums are fwd_tile's (sigma_half's rounding, the
// same alpha test, the cut's compare without opacities); a pixel that fails
// the test adds zeros, so the walk has no branches.  A chunk with a record
// that could make those zeros NaN (no culling data under TAME packing) takes a
// scalar walk that skips failing pixels.
// Bound by the FMA pipe and issue together (66% of the cycles and of the slots; a
// packed operation takes two cycles of the FMA pipe, so packing saves issue slots
// only).  2048^2 / 1M Gaussians: 973 us, against 1265 with one pixel a lane in
// 8x4 regions (scalar, skipping); 8x16 regions with two pairs a lane: 1120 (fewer operations a
// pixel, more pixels out of reach).
struct GaAcc {
    // colour, wsum; sums of c alpha sx, c alpha sy (negated when written) and
    // c alpha (sx sy - b)
    f2 c[3], w, x[3], y[3], xy[3];
    int cur[2];
};

__device__ __forceinline__ f2 f2_add_half(f2 v, int h, float x) {
    float lo, hi;
    f2_unpack(v, lo, hi);
    return h ? f2_pack(lo, hi + x) : f2_pack(lo + x, hi);
}

template <bool OP>
__device__ __forceinline__ void ga_walk(uint32_t mask, const Rec<float> *rb, int ib, float px,
                                        f2 py, uint32_t cut, GaAcc &A) {
    const f2 HALF = f2_dup(0.5f);
    while (mask) {
        const int bit = __ffs(mask) - 1;
        mask &= mask - 1;
        const Rec<float> &g = rb[bit];
        const float4 q0 = *reinterpret_cast<const float4 *>(&g.x);
        const float4 q1 = *reinterpret_cast<const float4 *>(&g.c);
        // sigma and the slopes' products are even in d, so d = pixel - mean
        // gives fwd_tile's values
        const f2 DX = f2_dup(px - q0.x), DY = f2_add(py, f2_dup(-q0.y));
        const f2 B = f2_dup(q0.w), C = f2_dup(q1.x);
        const f2 AX = f2_mul(f2_dup(q0.z), DX), BX = f2_mul(B, DX);
        const f2 S = f2_fma(BX, DY, f2_fma(f2_mul(HALF, AX), DX,
                                           f2_mul(f2_mul(f2_mul(HALF, C), DY), DY)));
        float s0, s1;
        f2_unpack(S, s0, s1);
        float e0 = __expf(-s0), e1 = __expf(-s1);
        if constexpr (OP) {
            const float o = g.o;
            e0 *= o;
            e1 *= o;
        }
        float a0 = fminf(0.999f, e0), a1 = fminf(0.999f, e1);
        bool no0, no1;
        if constexpr (!OP && LIG_RASTER_ALPHA_CUT) {
            no0 = __float_as_uint(s0) >= cut;
            no1 = __float_as_uint(s1) >= cut;
        } else {
            no0 = s0 < 0.f || a0 < 1.f / 255.f;
            no1 = s1 < 0.f || a1 < 1.f / 255.f;
        }
        const f2 AL = f2_pack(no0 ? 0.f : a0, no1 ? 0.f : a1);
        A.cur[0] = no0 ? A.cur[0] : ib + bit;
        A.cur[1] = no1 ? A.cur[1] : ib + bit;
        const f2 SX = f2_fma(B, DY, AX), SY = f2_fma(C, DY, BX);
        const f2 WX = f2_mul(AL, SX), WY = f2_mul(AL, SY);
        const f2 WP = f2_mul(AL, f2_fma(SX, SY, f2_dup(-q0.w)));
        const f2 col[3] = {f2_dup(q1.y), f2_dup(q1.z), f2_dup(q1.w)};
        A.w = f2_add(A.w, AL);
#pragma unroll
        for (int ch = 0; ch < 3; ++ch) {
            A.c[ch] = f2_fma(col[ch], AL, A.c[ch]);
            A.x[ch] = f2_fma(col[ch], WX, A.x[ch]);
            A.y[ch] = f2_fma(col[ch], WY, A.y[ch]);
            A.xy[ch] = f2_fma(col[ch], WP, A.xy[ch]);
        }
    }
}

// The same chunk pixel by pixel, skipping what fails the alpha test.
__device__ __noinline__ void ga_walk_skip(uint32_t mask, const Rec<float> *rb, int ib, float px,
                                          float py0, GaAcc &A) {
    while (mask) {
        const int bit = __ffs(mask) - 1;
        mask &= mask - 1;
        const Rec<float> g = rb[bit];
        for (int h = 0; h < 2; ++h) {
            float dx, dy, a;
            if (!PixelEval<float>::alpha(g, px, py0 + (float)(4 * h), dx, dy, a))
                continue;
            const float sx = g.a * dx + g.b * dy, sy = g.b * dx + g.c * dy;
            const float wx = a * sx, wy = a * sy, wp = a * (sx * sy - g.b);
            const float c[3] = {g.r, g.g, g.bl};
#pragma unroll
            for (int ch = 0; ch < 3; ++ch) {
                A.c[ch] = f2_add_half(A.c[ch], h, c[ch] * a);
                A.x[ch] = f2_add_half(A.x[ch], h, c[ch] * wx);
                A.y[ch] = f2_add_half(A.y[ch], h, c[ch] * wy);
                A.xy[ch] = f2_add_half(A.xy[ch], h, c[ch] * wp);
            }
            A.w = f2_add_half(A.w, h, a);
            A.cur[h] = ib + bit;
        }
    }
}

template <bool OP, int MAXT, int MINB>
__global__ void __launch_bounds__(MAXT, MINB)
raster_fwd_ga_kernel(const BatchGeo geo, const int32_t *__restrict__ cum, int *work,
                     const int32_t *__restrict__ ids, const int2 *__restrict__ tile_bins,
                     const int32_t *__restrict__ d_total, const Rec<float> *__restrict__ recs,
                     float *__restrict__ img, float *__restrict__ wsum, float *__restrict__ odx,
                     float *__restrict__ ody, float *__restrict__ odxy,
                     int32_t *__restrict__ final_idx) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ int s_slot;
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    Rec<float> *w_rec = reinterpret_cast<Rec<float> *>(smem_raw) + w * 32;
    const int n_tiles = geo.total_tiles();
    const uint32_t cut = OP ? 0u : g_alpha_cut;
    for (int tile = next_tile(work, s_slot, true); tile < n_tiles;
         tile = next_tile(work, s_slot, false)) {
        const TileCtx tc = tile_ctx(geo, cum, d_total, tile);
        const Regions R = Regions::make(1, tc.B);
        int lx, ly;
        R.pixel(w, lane, 0, lx, ly);
        const int gx = tc.tx0 + lx, gy = tc.ty0 + ly;
        const float px = (float)gx + 0.5f, py = (float)gy + 0.5f;
        const f2 py2 = f2_pack(py, (float)(gy + 4) + 0.5f);
        GaAcc A;
        A.w = f2_zero();
        A.cur[0] = A.cur[1] = 0;
#pragma unroll
        for (int ch = 0; ch < 3; ++ch) A.c[ch] = A.x[ch] = A.y[ch] = A.xy[ch] = f2_zero();
        if (!tc.empty) {
            const int2 range = tile_bins[tile];
            Rec<float> pre;
            if (range.x + lane < range.y) pre = recs[__ldg(ids + range.x + lane)];
            for (int base = range.x; base < range.y; base += 32) {
                const bool mine = base + lane < range.y;
                const bool hit = mine && region_hit<float, true, false>(pre, R, w, tc.tx0, tc.ty0);
                const bool fast = !__any_sync(FULL, mine && !(pre.wx >= 0.f));
                __syncwarp();
                w_rec[lane] = pre;
                __syncwarp();
                if (base + 32 + lane < range.y) pre = recs[__ldg(ids + base + 32 + lane)];
                const uint32_t mask = __ballot_sync(FULL, hit);
                if (fast) {
                    ga_walk<OP>(mask, w_rec, base, px, py2, cut, A);
                } else {  // through a copy, so that A itself stays in registers
                    GaAcc t = A;
                    ga_walk_skip(mask, w_rec, base, px, py, t);
                    A = t;
                }
            }
        } else {  // the reference's empty-list branch (rasterize.py:80-90)
#pragma unroll
            for (int ch = 0; ch < 3; ++ch) A.c[ch] = f2_dup(1.f);
        }
        float v[2][13];
        f2_unpack(A.w, v[0][12], v[1][12]);
#pragma unroll
        for (int ch = 0; ch < 3; ++ch) {
            f2_unpack(A.c[ch], v[0][ch], v[1][ch]);
            f2_unpack(A.x[ch], v[0][3 + ch], v[1][3 + ch]);
            f2_unpack(A.y[ch], v[0][6 + ch], v[1][6 + ch]);
            f2_unpack(A.xy[ch], v[0][9 + ch], v[1][9 + ch]);
        }
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            if (!(lx < tc.B && ly + 4 * h < tc.B && gx < tc.W && gy + 4 * h < tc.H)) continue;
            const int pix = tc.poff + (gy + 4 * h) * tc.W + gx;
            final_idx[pix] = A.cur[h];
            wsum[pix] = v[h][12];
#pragma unroll
            for (int ch = 0; ch < 3; ++ch) {
                img[3 * pix + ch] = v[h][ch];
                odx[3 * pix + ch] = 0.f - v[h][3 + ch];
                ody[3 * pix + ch] = 0.f - v[h][6 + ch];
                odxy[3 * pix + ch] = v[h][9 + ch];
            }
        }
    }
}

// Loss from the tile partials, deterministic, in one launch.  Each CTA sums a
// chunk of kLossChunk tile partials of one image (thread-strided, then a
// fixed-order block reduction); image i owns CTAs [chunk_off[i],
// chunk_off[i+1]).  The CTA that finishes last (a ticket, cleared by this
// call's pack) adds every image's chunk sums in order (a warp per image,
// lane-strided + butterfly), divides by 3 H_i W_i and adds the image means in
// order; whichever CTA that is, the sums are the same.  In the fit step one more
// CTA forms Adam's scalars meanwhile.
// Latency-bound: 2048^2 6 us with chunks of 1024 tiles (4096 and a second launch:
// 12), 512^2 4.6 (5 and a launch gap).
constexpr int kLossChunk = 1024;

struct TileChunks {
    int n_img;
    int chunk_off[kMaxBatch + 1];
};

// Tile partials, then the chunk sums (at most one per kLossChunk tiles plus one
// per image of a batch), then the loss kernel's ticket.
inline size_t loss_ticket_offset(int num_tiles) {
    const size_t t = (size_t)(num_tiles > 0 ? num_tiles : 0);
    return t + t / kLossChunk + 1 + kMaxBatch;
}
inline uint32_t *loss_ticket(double *partials, int num_tiles) {
    return reinterpret_cast<uint32_t *>(partials + loss_ticket_offset(num_tiles));
}

inline TileChunks tile_chunks(const BatchGeo &geo) {
    TileChunks c;
    c.n_img = geo.n_img;
    c.chunk_off[0] = 0;
    for (int i = 0; i < geo.n_img; ++i) {
        const int t = geo.tile_off[i + 1] - geo.tile_off[i];
        c.chunk_off[i + 1] = c.chunk_off[i] + (t + kLossChunk - 1) / kLossChunk;
    }
    return c;
}

template <typename T>
__global__ void __launch_bounds__(256)
l2_loss_kernel(const BatchGeo geo, const TileChunks ch, const double *__restrict__ partial,
               double *chunk_sum, uint32_t *ticket, T *__restrict__ loss,
               T *__restrict__ per_image, const AdamPro pro) {
    __shared__ double s_w[8], s_mean[kMaxBatch];
    __shared__ bool s_last;
    const int b = blockIdx.x, chunks = ch.chunk_off[ch.n_img];
    if (b == chunks) {
        fit_prologue(pro, geo.n_img);
        return;
    }
    const int im0 = BatchGeo::find(ch.chunk_off, ch.n_img, b);
    const int k0 = geo.tile_off[im0] + (b - ch.chunk_off[im0]) * kLossChunk;
    const int k1 = min(k0 + kLossChunk, geo.tile_off[im0 + 1]);
    double t = 0;
#pragma unroll 4
    for (int k = k0 + threadIdx.x; k < k1; k += blockDim.x) t += partial[k];
#pragma unroll
    for (int o = 16; o >= 1; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) s_w[w] = t;
    __syncthreads();
    if (threadIdx.x == 0) {
        double u = 0;
        for (int k = 0; k < (int)(blockDim.x >> 5); ++k) u += s_w[k];
        chunk_sum[b] = u;
        __threadfence();  // the sum before the ticket
        s_last = atomicAdd(ticket, 1u) == (uint32_t)chunks - 1;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();  // the ticket before the others' sums
    for (int im = w; im < geo.n_img; im += (int)(blockDim.x >> 5)) {
        double u = 0;
        for (int k = ch.chunk_off[im] + lane; k < ch.chunk_off[im + 1]; k += 32)
            u += __ldcg(chunk_sum + k);
#pragma unroll
        for (int o = 16; o >= 1; o >>= 1) u += __shfl_xor_sync(0xffffffffu, u, o);
        if (lane == 0) {
            const double m = u / (3.0 * (double)geo.H[im] * (double)geo.W[im]);
            s_mean[im] = m;
            if (per_image) per_image[im] = (T)m;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double total = 0;
        for (int im = 0; im < geo.n_img; ++im) total += s_mean[im];
        *loss = (T)total;
    }
}

// ------------------------------------------------------------- backward
template <typename T>
struct Grads {  // the ABI's per-Gaussian gradient arrays (v_opac may be null)
    T *v_xy, *v_abs, *v_conic, *v_rgb, *v_opac;
};

// Backward, transposed: one CTA per tile, warp w owns region w (an 8x4 block in
// the sum variant; in the gradient-aware variant the reference's warp w, whose
// v_xy_abs is |sum over that warp| per Gaussian,
// csrc/gradient_aware_rasterizer.cu:317-341).  The tile's pixel cotangents,
// pixel centres and final indices are staged in shared memory once, region
// by region.  Per batch each warp compacts the batch slots whose region box it
// meets (exact ellipse test by the lanes); lanes then take one such Gaussian
// each — or, for a short list, 2 / 4 / 8 lanes share one and take interleaved
// pixels — and loop over the region's pixels (pixel data read by broadcast),
// accumulating the Gaussian's gradient terms in registers; a lane group is
// combined with shuffles, and the terms go to the packed per-Gaussian buffer
// with 16-byte atomics per (Gaussian, region) — [N][12], three atomics, in
// general; [N][8], two, in the lean fused-loss variant.  Entries past every
// pixel's final index are skipped.
//
// Pixel cotangent source of the backward: explicit dL/dimg (+ optional
// dL/dwsum), or — fused L2 — computed on the fly from the render and the target
// as the gradient of mean((clamp(img, 0, 1) - target)^2): the value torch's
// mse_loss + clamp backward produce, 2/N (clamp(x) - t) g where 0 <= x <= 1.
template <typename T>
struct CotSrc {
    const T *v_img, *v_wsum;              // explicit (v_wsum may be null: zero)
    const T *img, *target, *grad_loss;    // fused L2 (v_img == null)
    T scale;                              // 2 / numel
    const T *diff = nullptr;              // fused L2 from the forward's masked difference
    __device__ __forceinline__ void get(int p, T &r, T &g, T &b, T &w) const {
        w = v_wsum ? v_wsum[p] : (T)0;
        if (v_img) {
            r = v_img[3 * p];
            g = v_img[3 * p + 1];
            b = v_img[3 * p + 2];
            return;
        }
        const T s = scale * *grad_loss;
        if (diff) {
            r = diff[3 * p] * s;
            g = diff[3 * p + 1] * s;
            b = diff[3 * p + 2] * s;
            return;
        }
        T v[3];
#pragma unroll
        for (int ch = 0; ch < 3; ++ch) {
            const T x = img[3 * p + ch];
            const T d = min(max(x, (T)0), (T)1) - target[3 * p + ch];
            v[ch] = (x >= (T)0 && x <= (T)1) ? d * s : (T)0;
        }
        r = v[0]; g = v[1]; b = v[2];
    }
};

template <typename T, bool GA>
struct alignas(16) PixRec {
    T vo0, vo1, vo2, vw;  // first: one 16-byte load in the lean loop
    T px, py;
    int fin;
    T vd[GA ? 9 : 1];  // vdx.rgb, vdy.rgb, vdxy.rgb
};

#ifndef LIG_RASTER_BWD_COLS
#define LIG_RASTER_BWD_COLS 1  // lean backward: column-major region walk
#endif

// Lean backward of one Gaussian over the pixels of one 8x4 region that this
// lane takes: columns part, part + 2^LS, ... (8 >> LS of them) in each of the
// four rows, column by column.  The separable pieces of sigma are shared:
// per row dy and (c/2 dy) dy, per column dx, (a/2) dx and b dx, so that
//   sigma = fma(b dx, dy, fma((a/2) dx, dx, ((c/2) dy) dy))
// which equals sigma_ref's fma(b dx, dy, 0.5 fma(a dx, dx, (c dy) dy)) bit for
// bit (halving is exact and commutes with rounding away from the subnormal
// range) with one product fewer.  No opacities on this path (o = 1, so
// alpha = min(clamp, exp(-sigma)) is the reference's o * exp(-sigma) clamped).
// No final-index test either: a Gaussian after a pixel's final index fails
// that pixel's alpha test here exactly as it did in the forward.  A skipped
// pair adds zeros.  The moment sums of v_sigma dx^i dy^j (v_sigma =
// -alpha v_alpha) use dx constant along a column: Sx, Sxx and Sxy take one
// term per column.  Leaves Sx, Sy, Sxx, Sxy, Syy in acc[0, 1, 4, 5, 6] and the
// colour sums in acc[7..9].
template <typename T, int LS>
__device__ __forceinline__ void lean_region(const Rec<T> &g, T clamp,
                                            const PixRec<T, false> *__restrict__ pix, int part,
                                            T px0, T py0, T (&acc)[11]) {
    using M = Math<T>;
    constexpr int NC = 8 >> LS, JS = 1 << LS;
    const T ha = (T)0.5 * g.a, hc = (T)0.5 * g.c;
    T dy[4], cdd[4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        dy[r] = g.y - (py0 + (T)r);
        cdd[r] = mul_rn(mul_rn(hc, dy[r]), dy[r]);
    }
    T sx = 0, sy = 0, sxx = 0, sxy = 0, syy = 0, c0 = 0, c1 = 0, c2 = 0;
#pragma unroll
    for (int k = 0; k < NC; ++k) {
        const T dx = g.x - (px0 + (T)(k * JS));
        const T hadx = mul_rn(ha, dx), bdx = mul_rn(g.b, dx);
        T wc = 0, yc = 0;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const PixRec<T, false> &c = pix[r * 8 + part + k * JS];
            const T s = fma_rn(bdx, dy[r], fma_rn(hadx, dx, cdd[r]));
            const T al = M::min_(clamp, M::exp_(-s));
            const T a = (s < (T)0 || al < (T)1 / (T)255) ? (T)0 : al;
            c0 += a * c.vo0;
            c1 += a * c.vo1;
            c2 += a * c.vo2;
            const T wv = a * (g.r * c.vo0 + g.g * c.vo1 + g.bl * c.vo2);  // -v_sigma
            wc += wv;
            const T ty = wv * dy[r];
            yc += ty;
            syy += ty * dy[r];
        }
        const T tx = wc * dx;
        sx += tx;
        sxx += tx * dx;
        sy += yc;
        sxy += yc * dx;
    }
    acc[0] = -sx; acc[1] = -sy; acc[4] = -sxx; acc[5] = -sxy; acc[6] = -syy;
    acc[7] = c0; acc[8] = c1; acc[9] = c2;
}

#ifndef LIG_RASTER_BWD_F2
#define LIG_RASTER_BWD_F2 1  // lean backward (float): pixel pairs in f32x2 arithmetic
#endif

// The lean backward's pixel cotangents in pair layout: region entry
// row * 4 + cp holds columns cp and cp + 4 of that row, channel by channel,
// so one 16-byte and one 8-byte load give three ready (column cp, cp + 4)
// pairs.
struct alignas(16) PixPair {
    float v[8];  // v0 (cp, cp+4), v1 (cp, cp+4), v2 (cp, cp+4), v_wsum (GEN walks)
};

// lean_region in f32x2 form (float): the lane takes NCP column pairs
// c0, c0 + CSTEP, ... (columns cp and cp + 4 of each) in NR rows r0.. of the
// 8-column region, and evaluates the two pixels of a pair with one packed
// operation where lean_region uses two.  Per pixel the operations and their
// roundings are lean_region's — sigma = fma(b dx, dy, fma((a/2) dx, dx,
// ((c/2) dy) dy)), alpha = min(clamp, exp(-sigma)) and the same alpha test —
// so the alpha decisions are bit-identical; only the order in which the
// moment and colour sums are added differs.  Same quantities as lean_region,
// added to acc[] (zeroed by the caller).  NH > 1 walks NH blocks of NR rows
// (rows r0 .. r0 + NH NR - 1 of a taller region, 4 pair entries a row in pp).
// ABS: also the per-pixel absolute values of the mean gradient summed over
// the pixels (the reference's v_xy_abs, csrc/backward.cu:146-150), in acc[2],
// acc[3]: per pixel v_sigma (a dx + b dy) and v_sigma (b dx + c dy).
// GEN: opacities and a wsum cotangent (pair entry's fourth channel); the
// opacity gradient's sum of exp(-sigma) v_alpha in acc[10].
template <int NCP, int CSTEP, int NR, bool ABS = false, int NH = 1, bool GEN = false,
          bool CUT = false>
__device__ __forceinline__ void lean_region_f2(const Rec<float> &g, float clamp,
                                               const PixPair *__restrict__ pp, int c0, int r0,
                                               float px0, float py0, uint32_t cut,
                                               float (&acc)[11]) {
    const float ha = g.a, hc = g.c;  // the record's halved conic
    const f2 HA = f2_dup(ha), BB = f2_dup(g.b);
    f2 AA, CC;
    float ax = 0.f, ay = 0.f;
    if constexpr (ABS) {
        AA = f2_dup(2.f * ha);
        CC = f2_dup(2.f * hc);
    }
    const f2 CR = f2_dup(g.r), CG = f2_dup(g.g), CB = f2_dup(g.bl);
    f2 sx = f2_zero(), sy = f2_zero(), sxx = f2_zero(), sxy = f2_zero(), syy = f2_zero();
    f2 sr = f2_zero(), sg = f2_zero(), sb = f2_zero();
    [[maybe_unused]] f2 so = f2_zero();
    // NH blocks of NR rows, one after the other (not interleaved: the sums
    // carry over, the row and column products are rebuilt per block)
#pragma unroll 1
    for (int hh = 0; hh < NH; ++hh) {
        const int rb = r0 + hh * NR;
        f2 DY[NR], CDD[NR];
#pragma unroll
        for (int r = 0; r < NR; ++r) {
            const float dy = g.y - (py0 + (float)(rb + r));
            DY[r] = f2_dup(dy);
            CDD[r] = f2_dup(__fmul_rn(__fmul_rn(hc, dy), dy));
        }
#pragma unroll
        for (int k = 0; k < NCP; ++k) {
            const int cp = c0 + k * CSTEP;
            const f2 DX = f2_pack(g.x - (px0 + (float)cp), g.x - (px0 + (float)(cp + 4)));
            const f2 HADX = f2_mul(HA, DX), BDX = f2_mul(BB, DX);
            f2 AX;
            if constexpr (ABS) AX = f2_mul(AA, DX);
            f2 wc = f2_zero(), yc = f2_zero();
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                const PixPair *e = pp + (rb + r) * 4 + cp;
                const ulonglong2 v01 = *reinterpret_cast<const ulonglong2 *>(e->v);
                const f2 V0{v01.x}, V1{v01.y};
                const f2 V2{*reinterpret_cast<const unsigned long long *>(e->v + 4)};
                const f2 S = f2_fma(BDX, DY[r], f2_fma(HADX, DX, CDD[r]));
                float s0, s1;
                f2_unpack(S, s0, s1);
                const float vis0 = __expf(-s0), vis1 = __expf(-s1);
                const float al0 = fminf(clamp, GEN ? g.o * vis0 : vis0);
                const float al1 = fminf(clamp, GEN ? g.o * vis1 : vis1);
                const bool no0 = CUT ? __float_as_uint(s0) >= cut : s0 < 0.f || al0 < 1.f / 255.f;
                const bool no1 = CUT ? __float_as_uint(s1) >= cut : s1 < 0.f || al1 < 1.f / 255.f;
                const f2 A = f2_pack(no0 ? 0.f : al0, no1 ? 0.f : al1);
                sr = f2_fma(A, V0, sr);
                sg = f2_fma(A, V1, sg);
                sb = f2_fma(A, V2, sb);
                // -v_sigma per pixel
                f2 VA = f2_fma(CB, V2, f2_fma(CG, V1, f2_mul(CR, V0)));
                if constexpr (GEN) {
                    VA = f2_add(VA, f2{*reinterpret_cast<const unsigned long long *>(e->v + 6)});
                    so = f2_fma(f2_pack(no0 ? 0.f : vis0, no1 ? 0.f : vis1), VA, so);
                }
                const f2 WV = f2_mul(A, VA);
                wc = f2_add(wc, WV);
                const f2 TY = f2_mul(WV, DY[r]);
                yc = f2_add(yc, TY);
                syy = f2_fma(TY, DY[r], syy);
                if constexpr (ABS) {
                    float gx0, gx1, gy0, gy1;
                    f2_unpack(f2_mul(WV, f2_fma(BB, DY[r], AX)), gx0, gx1);
                    f2_unpack(f2_mul(WV, f2_fma(CC, DY[r], BDX)), gy0, gy1);
                    ax += fabsf(gx0) + fabsf(gx1);
                    ay += fabsf(gy0) + fabsf(gy1);
                }
            }
            const f2 TX = f2_mul(wc, DX);
            sx = f2_add(sx, TX);
            sxx = f2_fma(TX, DX, sxx);
            sy = f2_add(sy, yc);
            sxy = f2_fma(yc, DX, sxy);
        }
    }
    acc[0] -= f2_sum(sx); acc[1] -= f2_sum(sy);
    acc[4] -= f2_sum(sxx); acc[5] -= f2_sum(sxy); acc[6] -= f2_sum(syy);
    acc[7] += f2_sum(sr); acc[8] += f2_sum(sg); acc[9] += f2_sum(sb);
    if constexpr (ABS) {
        acc[2] += ax;
        acc[3] += ay;
    }
    if constexpr (GEN) acc[10] += f2_sum(so);
}

// GEN walks: one Gaussian over the region's pixels part, part + step, ... one
// at a time (row-major 8-column region at pixel (rx, ry)), skipping what fails
// the alpha test or lies outside: records and tiles whose zeros could turn
// into NaN.  csrc/backward.cu:102-150; leaves the gradients themselves (no
// moments) in acc.
__device__ __noinline__ void sum_pixels_skip(const Rec<float> &half, float clamp,
                                             const PixPair *pp, int npix, int part, int step,
                                             int rx, int ry, int x_end, int y_end, float *acc) {
    Rec<float> g = half;
    g.a *= 2.f;
    g.c *= 2.f;
    for (int j = part; j < npix; j += step) {
        const int row = j >> 3, col = j & 7, h = col >> 2;
        if (rx + col >= x_end || ry + row >= y_end) continue;
        const float *v = pp[row * 4 + (col & 3)].v;
        const float dx = g.x - ((float)(rx + col) + 0.5f), dy = g.y - ((float)(ry + row) + 0.5f);
        const float sigma = sigma_ref<float>(g.a, g.b, g.c, dx, dy);
        const float vis = __expf(-sigma);
        const float alpha = fminf(clamp, g.o * vis);
        if (sigma < 0.f || alpha < 1.f / 255.f) continue;
        acc[7] += alpha * v[h];
        acc[8] += alpha * v[2 + h];
        acc[9] += alpha * v[4 + h];
        float v_alpha = 0.f;
        v_alpha += g.r * v[h];
        v_alpha += g.g * v[2 + h];
        v_alpha += g.bl * v[4 + h];
        v_alpha += v[6 + h];
        acc[10] += vis * v_alpha;
        const float v_sigma = -alpha * v_alpha;
        acc[4] += 0.5f * v_sigma * dx * dx;
        acc[5] += v_sigma * dx * dy;
        acc[6] += 0.5f * v_sigma * dy * dy;
        const float gx = v_sigma * (g.a * dx + g.b * dy), gy = v_sigma * (g.b * dx + g.c * dy);
        acc[0] += gx;
        acc[1] += gy;
        acc[2] += fabsf(gx);
        acc[3] += fabsf(gy);
    }
}

// Lean walks: the alpha cut's compare (one operation of the half-rate ALU pipe
// instead of two per pixel) where every Gaussian of a warp's round has culling
// data.  8192^2 1992 -> 1891 us, 2048^2 / 1M 747 -> 705 (681 at 7 CTAs
// per SM), 16 images 402 -> 371.
#ifndef LIG_RASTER_BWD_CUT
#define LIG_RASTER_BWD_CUT 1
#endif
#ifndef LIG_RASTER_BWD_BULK
#define LIG_RASTER_BWD_BULK 1  // lean backward (float): records staged by bulk async copies
#endif
// One lane's share of a Gaussian over its region, in blocks of four rows: 1 / 2 /
// 4 / 8 lanes (lsplit) share the Gaussian, taking column pairs (1 / 2 / 4 lanes)
// or column pairs and row halves (8 lanes).
template <int RR, bool ABS, bool GEN, bool CUT>
__device__ __forceinline__ void lean_round(const Rec<float> &g, float clamp,
                                           const PixPair *__restrict__ pp, int lsplit, int part,
                                           float px0, float py0, uint32_t cut, float (&acc)[11]) {
    constexpr int NB = RR / 4;
    switch (lsplit) {
    case 0:
        lean_region_f2<4, 1, 4, ABS, NB, GEN, CUT>(g, clamp, pp, 0, 0, px0, py0, cut, acc);
        break;
    case 1:
        lean_region_f2<2, 2, 4, ABS, NB, GEN, CUT>(g, clamp, pp, part, 0, px0, py0, cut, acc);
        break;
    case 2:
        lean_region_f2<1, 1, 4, ABS, NB, GEN, CUT>(g, clamp, pp, part, 0, px0, py0, cut, acc);
        break;
    default:
        if constexpr (RR == 4)
            lean_region_f2<1, 1, 2, ABS, 1, GEN, CUT>(g, clamp, pp, part & 3, 2 * (part >> 2), px0,
                                                      py0, cut, acc);
        else
            lean_region_f2<1, 1, 4, ABS, NB / 2, GEN, CUT>(g, clamp, pp, part & 3,
                                                           (RR / 2) * (part >> 2), px0, py0, cut,
                                                           acc);
        break;
    }
}

// Bounded device waits that gave up (a malfunction; read by lig_wait_timeouts).
__device__ unsigned int g_wait_timeouts;
// SM clock cycles (about 1 ms) before an mbarrier wait is abandoned: a
// normal wait ends within microseconds, and a malfunction then costs a
// launch at most about a millisecond per wave of CTAs instead of a hang.
constexpr long long kWaitCycles = 2000000;

// Bulk asynchronous copies of gathered 48-byte records into shared memory,
// completing on one mbarrier per CTA (cp.async.bulk, this GPU's memory only,
// no multicast).  Thread 0 announces the batch's bytes; each thread < cnt
// copies its record.  The transaction count may be completed before it is
// announced (its range includes negative values), so no barrier is needed
// between the two.
__device__ __forceinline__ void bulk_records(uint32_t bar, Rec<float> *s_rec, int32_t *s_ids,
                                             const int32_t *__restrict__ ids,
                                             const Rec<float> *__restrict__ recs, int base,
                                             int cnt) {
    const int tid = threadIdx.x;
    if (tid == 0)
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar),
                     "r"(cnt * (int)sizeof(Rec<float>))
                     : "memory");
    if (tid < cnt) {
        const int id = __ldg(ids + base + tid);
        s_ids[tid] = id;
        const uint32_t dst = (uint32_t)__cvta_generic_to_shared(s_rec + tid);
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, "
            "[%3];" ::"r"(dst),
            "l"(recs + id), "r"((int)sizeof(Rec<float>)), "r"(bar)
            : "memory");
    }
}

// Wait for the mbarrier's phase `phase` for at most kWaitCycles.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t phase) {
    uint32_t done = 0;
    const long long t0 = clock64();
    for (;;) {
        asm volatile(
            "{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; "
            "selp.u32 %0, 1, 0, p; }"
            : "=r"(done)
            : "r"(bar), "r"(phase)
            : "memory");
        if (done || clock64() - t0 > kWaitCycles) break;
    }
    return done != 0;
}

// Pair walks read records with the halved conic (a/2, c/2; see sigma_half).
// LEAN (sum backward of the fused fit loss, no opacities, no wsum
// cotangent): only the gradients the fit needs — v_xy, v_conic, v_rgb — are
// accumulated (no |v_xy| sums, no opacity gradient) and each (Gaussian,
// region) pair adds them with two 16-byte atomics into an [N][8] buffer.
// RR (float pair walk only): region rows, 4 (8x4 regions, eight warps per
// 16x16 tile), 8 (8x8, four warps, each thread staging two pixels) or 16
// (8x16, two warps, four pixels a thread); a lane group walks a taller region
// in blocks of four rows.
// Against 8x4 regions a Gaussian meets fewer regions, so the per-pair costs —
// the warps' region tests, the per-round set-up, the lane-group reduction and
// the atomics — are paid fewer times, for more pixel evaluations per pair.
// GEN (with ABS): opacities and a wsum cotangent in the pair walk, where an
// opacity costs a product and a multiply-add a pixel; bound by the FMA pipe and
// issue as the lean walk.  Records
// without culling data (under TAME packing) and tiles with a cotangent above
// kTameCot or non-finite take sum_pixels_skip.
template <typename T, bool GA, bool LEAN, bool ABS = false, int RR = 4, bool GEN = false>
__device__ __forceinline__ void bwd_tile(const TileCtx &tc, int tile,
                                         const int32_t *__restrict__ ids,
                                         const int2 *__restrict__ tile_bins,
                                         const Rec<T> *__restrict__ recs,
                                         const int32_t *__restrict__ final_idx, CotSrc<T> cot,
                                         const T *__restrict__ v_dx, const T *__restrict__ v_dy,
                                         const T *__restrict__ v_dxy, T clamp,
                                         T *__restrict__ packed, int &s_end, uint32_t bar,
                                         uint32_t &phase) {
    using M = Math<T>;
    // float lean backward: pixel pairs in f32x2 arithmetic (lean_region_f2)
    constexpr bool kPairs = LEAN && !GA && LIG_RASTER_BWD_F2 && sizeof(T) == 4;
    static_assert(!ABS || kPairs, "the |v_xy| sums of the lean walk need its pair form");
    static_assert(!GEN || ABS, "the general pair walk keeps the |v_xy| sums");
    [[maybe_unused]] bool tame_cot = true;
    // records staged by bulk async copies (no register prefetch, no region
    // masks: the warps test the box and ellipse themselves)
    constexpr bool kBulk = kPairs && LIG_RASTER_BWD_BULK;
    constexpr bool kCut = kPairs && !GEN && LIG_RASTER_BWD_CUT;
    [[maybe_unused]] const uint32_t cut = kCut ? g_alpha_cut : 0u;
    static_assert(RR == 4 || kPairs, "taller regions are walked by the pair form only");
    static_assert(RR == 4 || RR == 8 || RR == 16, "region rows");
    constexpr int kRows = RR;  // pair entries per region: kRows * 4
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int nt = blockDim.x;  // = 32 * regions: region-major pixel slots
    PixRec<T, GA> *s_pix = reinterpret_cast<PixRec<T, GA> *>(smem_raw);
    // (8x16 regions: two pixel slots a thread hold the pair entries)
    Rec<T> *s_rec = reinterpret_cast<Rec<T> *>(s_pix + nt * (RR == 16 ? 2 : 1));
    uint32_t *s_bits = reinterpret_cast<uint32_t *>(s_rec + nt);
    int32_t *s_ids = reinterpret_cast<int32_t *>(s_bits + nt);
    uint16_t *s_list = reinterpret_cast<uint16_t *>(s_ids + nt);
    const unsigned FULL = 0xffffffffu;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    if (tc.empty) return;  // gradients stay zero (rasterize.py:156-161)
    const int B = tc.B, H = tc.H, W = tc.W, tx0 = tc.tx0, ty0 = tc.ty0;
    // fused L2: mean over this image's 3HW values (a batch sums per-image means)
    if (!cot.v_img) cot.scale = (T)(2.0 / (3.0 * (double)H * (double)W));
    const Regions R = Regions::make(GA ? 2 : (RR == 8 ? 1 : RR == 16 ? 3 : 0), B);
    T rx0 = 0, rx1 = 0, ry0 = 0, ry1 = 0;  // this warp's region (tile-local centres)
    if (LIG_RASTER_BWD_LANE_ELLIPSE) R.rect<T>(w, rx0, rx1, ry0, ry1);
    uint16_t *my_list = s_list + w * nt;
    const PixRec<T, GA> *my_pix = s_pix + w * 32;

    const int2 range = tile_bins[tile];
    int end = range.y;
    Rec<T> pre;
    int pre_id = -1;
    if constexpr (kBulk) {
        // first batch in flight while the pixels are staged
        if (range.x < end)
            bulk_records(bar, reinterpret_cast<Rec<float> *>(s_rec), s_ids, ids,
                         reinterpret_cast<const Rec<float> *>(recs), range.x,
                         min(nt, end - range.x));
    } else if constexpr (LEAN) {
        // the lean walk has no final-index test (see lean_region), so the list
        // is not cut at the tile's last final index: the first batch's gather
        // is issued before the pixels are staged and no barrier precedes it
        if (range.x + tid < end) {
            pre_id = __ldg(ids + range.x + tid);
            pre = recs[pre_id];
        }
    }
    // stage this thread's pixel (region w, slot lane)
    if (!LEAN && tid == 0) s_end = -1;
    if constexpr (RR > 4) {
        // pixels (x, y + 4 p2) of region w; pair entries as below with RR rows
        // per region
#pragma unroll
        for (int p2 = 0; p2 < RR / 4; ++p2) {
            int lx, ly;
            R.pixel(w, lane, p2, lx, ly);
            const int gx = tx0 + lx, gy = ty0 + ly;
            const bool inside = lx < B && ly < B && gx < W && gy < H;
            T v0 = (T)0, v1 = (T)0, v2 = (T)0, vw = (T)0;
            if (inside) cot.get(tc.poff + gy * W + gx, v0, v1, v2, vw);
            PixPair *e = reinterpret_cast<PixPair *>(smem_raw) + w * RR * 4 +
                         ((lane >> 3) + 4 * p2) * 4 + (lane & 3);
            const int h = (lane >> 2) & 1;
            e->v[h] = v0;
            e->v[2 + h] = v1;
            e->v[4 + h] = v2;
            if constexpr (GEN) {
                e->v[6 + h] = vw;
                tame_cot = tame_cot && tame_cotangent(v0, v1, v2, vw);
            }
        }
    } else {
        int lx, ly;
        R.pixel(w, lane, 0, lx, ly);
        const int gx = tx0 + lx, gy = ty0 + ly;
        const bool inside = lx < B && ly < B && gx < W && gy < H;
        const int p = inside ? tc.poff + gy * W + gx : 0;
        PixRec<T, GA> c;
        c.px = (T)gx + (T)0.5;
        c.py = (T)gy + (T)0.5;
        c.vo0 = c.vo1 = c.vo2 = c.vw = (T)0;
        if (inside) cot.get(p, c.vo0, c.vo1, c.vo2, c.vw);
        c.fin = (!LEAN && inside) ? final_idx[p] : -1;  // -1: never valid (unread when lean)
        if constexpr (GA) {
#pragma unroll
            for (int ch = 0; ch < 3; ++ch) {
                c.vd[ch] = inside ? v_dx[3 * p + ch] : (T)0;
                c.vd[3 + ch] = inside ? v_dy[3 * p + ch] : (T)0;
                c.vd[6 + ch] = inside ? v_dxy[3 * p + ch] : (T)0;
            }
        }
        if constexpr (kPairs) {
            // region w's pair entries: (row, column) -> entry row * 4 + col % 4,
            // half col / 4 (the pixel slots are row-major 8x4, kind 0)
            PixPair *e = reinterpret_cast<PixPair *>(smem_raw) + w * 16 + (lane >> 3) * 4 +
                         (lane & 3);
            const int h = (lane >> 2) & 1;
            e->v[h] = c.vo0;
            e->v[2 + h] = c.vo1;
            e->v[4 + h] = c.vo2;
            if constexpr (GEN) {
                e->v[6 + h] = c.vw;
                tame_cot = tame_cotangent(c.vo0, c.vo1, c.vo2, c.vw);
            }
        } else {
            s_pix[tid] = c;
        }
        if constexpr (!LEAN) {
            int my_max = c.fin;
#pragma unroll
            for (int o = 16; o >= 1; o >>= 1)
                my_max = max(my_max, __shfl_xor_sync(FULL, my_max, o));
            __syncthreads();
            if (lane == 0) atomicMax(&s_end, my_max);
        }
    }
    if constexpr (!LEAN) {
        __syncthreads();
        end = min(range.y, s_end + 1);
        if (range.x + tid < end) {
            pre_id = __ldg(ids + range.x + tid);
            pre = recs[pre_id];
        }
    }
    [[maybe_unused]] bool wild = false;
    if constexpr (GEN) wild = __syncthreads_or(!tame_cot);
    for (int base = range.x; base < end; base += nt) {
        const int cnt = min(nt, end - base);
        if constexpr (kBulk) {
            if (base != range.x) {  // everyone is done with the previous batch
                __syncthreads();
                bulk_records(bar, reinterpret_cast<Rec<float> *>(s_rec), s_ids, ids,
                             reinterpret_cast<const Rec<float> *>(recs), base, cnt);
            }
            const bool ok = mbar_wait(bar, phase);
            phase ^= 1u;
            // all threads agree: a wait that gave up counts once, then every
            // thread lets its copies drain (bounded) and the tile is abandoned
            if (__syncthreads_or(!ok)) {
                if (tid == 0) atomicAdd(&g_wait_timeouts, 1u);
                (void)mbar_wait(bar, phase ^ 1u);
                return;
            }
        } else {
            __syncthreads();
            if (tid < cnt) {
                s_rec[tid] = pre;
                s_bits[tid] = region_bits<T, !LIG_RASTER_BWD_LANE_ELLIPSE>(pre, R, tx0, ty0);
                s_ids[tid] = pre_id;
            }
            __syncthreads();
            if (base + nt + tid < end) {
                pre_id = __ldg(ids + base + nt + tid);
                pre = recs[pre_id];
            }
        }
        // compact the batch slots touching this region (ascending)
        int nmine = 0;
        for (int m = 0; m * 32 < cnt; ++m) {
            const int t = m * 32 + lane;
            bool hit;
            if constexpr (kBulk) hit = t < cnt && region_hit<T, false, kPairs>(s_rec[t], R, w, tx0, ty0);
            else hit = t < cnt && ((s_bits[t] >> w) & 1u);
            if (LIG_RASTER_BWD_LANE_ELLIPSE && hit) {
                // exact ellipse test of Gaussian t against this warp's region,
                // one Gaussian per lane (the staging only tested the box)
                const Rec<T> &g = s_rec[t];
                if (g.wx >= (T)0) {
                    const T cx = g.x - (T)tx0, cy = g.y - (T)ty0;
                    const T a = kPairs ? (T)2 * g.a : g.a, c = kPairs ? (T)2 * g.c : g.c;
                    hit = !(sigma_min_rect<T>(a, g.b, c, rx0 - cx, rx1 - cx, ry0 - cy,
                                              ry1 - cy) > g.thr);
                }
            }
            const uint32_t mask = __ballot_sync(FULL, hit);
            if (hit) my_list[nmine + __popc(mask & ((1u << lane) - 1u))] = (uint16_t)t;
            nmine += __popc(mask);
        }
        __syncwarp();
        for (int g0 = 0, lsplit = 0; g0 < nmine; g0 += 32 >> lsplit) {
            // lanes per Gaussian: with at most LIG_RASTER_BWD_SPLIT3 / SPLIT2 /
            // SPLIT1 Gaussians left, 8 / 4 / 2 lanes share one Gaussian (a round
            // then takes 4 / 8 / 16 of them), lane part p taking pixels
            // p, p + 2^lsplit, ... of the region (interleaved, so the group's
            // pixel records sit in different shared-memory banks); their
            // sums are combined below
            const int left = min(32, nmine - g0);
            // (the 8x16 walk: its own first and last thresholds, 64-pixel
            // regions favour more lanes per Gaussian)
            constexpr int kS1 = RR == 16 ? LIG_RASTER_BWD_R16_SPLIT1 : LIG_RASTER_BWD_SPLIT1;
            constexpr int kS3 = RR == 16 ? LIG_RASTER_BWD_R16_SPLIT3 : LIG_RASTER_BWD_SPLIT3;
            lsplit = !LIG_RASTER_BWD_SPLIT             ? 0
                     : left <= kS3                     ? 3
                     : left <= LIG_RASTER_BWD_SPLIT2   ? 2
                     : left <= kS1                     ? 1 : 0;
            const int gi = lane >> lsplit, part = lane & ((1 << lsplit) - 1);
            const int jstep = 1 << lsplit;
            const int slot = gi < left ? (int)my_list[g0 + gi] : -1;
            const bool act = slot >= 0;
            const Rec<T> g = s_rec[act ? slot : 0];
            const int k = act ? base + slot : 0x7fffffff;
            T acc[11];
#pragma unroll
            for (int q = 0; q < 11; ++q) acc[q] = 0;
            bool touched = false;
            [[maybe_unused]] bool direct = false;  // acc holds gradients, not moments
            if constexpr (kPairs) {
                // as below, two pixels per packed operation: lanes of a group
                // take column pairs (1 / 2 / 4 lanes) or column pairs and row
                // halves (8 lanes)
                touched = act;
                const float px0 = (float)(tx0 + (w % R.nbx) * 8) + 0.5f;
                const float py0 = (float)(ty0 + (w / R.nbx) * kRows) + 0.5f;
                const PixPair *pp = reinterpret_cast<const PixPair *>(smem_raw) + w * kRows * 4;
                if constexpr (GEN) direct = act && (wild || !(g.wx >= (T)0));
                if (GEN && direct) {
                    float t[11] = {};
                    const int rx = tx0 + (w % R.nbx) * 8, ry = ty0 + (w / R.nbx) * kRows;
                    sum_pixels_skip(reinterpret_cast<const Rec<float> &>(s_rec[slot]), clamp, pp,
                                    kRows * 8, part, jstep, rx, ry, min(W, tx0 + B),
                                    min(H, ty0 + B), t);
#pragma unroll
                    for (int q = 0; q < 11; ++q) acc[q] = t[q];
                } else {
                    // the cut's compare where every Gaussian of the round has
                    // culling data (no opacities)
                    bool fast = false;
                    if constexpr (kCut)
                        fast = __all_sync(FULL, !act || reinterpret_cast<const Rec<float> &>(g).wx >= 0.f);
                    if (act) {
                        if (kCut && fast)
                            lean_round<RR, ABS, GEN, kCut>(g, clamp, pp, lsplit, part, px0, py0, cut, acc);
                        else
                            lean_round<RR, ABS, GEN, false>(g, clamp, pp, lsplit, part, px0, py0, cut, acc);
                    }
                }
            } else if constexpr (LEAN && !GA && LIG_RASTER_BWD_COLS) {
                // every listed (Gaussian, region) pair met the region's
                // ellipse test; an untouched one adds zeros
                touched = act;
                const T px0 = (T)(tx0 + (w % R.nbx) * 8 + part) + (T)0.5;
                const T py0 = (T)(ty0 + (w / R.nbx) * 4) + (T)0.5;
                if (act) {
                    switch (lsplit) {
                    case 0: lean_region<T, 0>(g, clamp, my_pix, part, px0, py0, acc); break;
                    case 1: lean_region<T, 1>(g, clamp, my_pix, part, px0, py0, acc); break;
                    case 2: lean_region<T, 2>(g, clamp, my_pix, part, px0, py0, acc); break;
                    default: lean_region<T, 3>(g, clamp, my_pix, part, px0, py0, acc); break;
                    }
                }
            } else {
            for (int j = part; j < 32; j += jstep) {
                const PixRec<T, GA> &c = my_pix[j];
                if (k > c.fin) continue;
                if constexpr (!GA) {
                    // csrc/backward.cu:102-150
                    const T dx = g.x - c.px;
                    const T dy = g.y - c.py;
                    const T sigma = sigma_ref<T>(g.a, g.b, g.c, dx, dy);
                    const T vis = M::exp_(-sigma);
                    const T alpha = M::min_(clamp, g.o * vis);
                    if (sigma < (T)0 || alpha < (T)1 / (T)255) continue;
                    touched = true;
                    T v_alpha = 0;
                    acc[7] += alpha * c.vo0;
                    acc[8] += alpha * c.vo1;
                    acc[9] += alpha * c.vo2;
                    v_alpha += g.r * c.vo0;
                    v_alpha += g.g * c.vo1;
                    v_alpha += g.bl * c.vo2;
                    if constexpr (!LEAN) {
                        v_alpha += c.vw;
                        acc[10] += vis * v_alpha;
                    }
                    const T v_sigma = -alpha * v_alpha;
                    if constexpr (LEAN) {
                        // the gradients are linear in five per-pixel sums
                        // (Sx, Sy, Sxx, Sxy, Syy of v_sigma dx^i dy^j); the
                        // conic is applied once per Gaussian after the loop
                        const T tx = v_sigma * dx, ty = v_sigma * dy;
                        acc[0] += tx;
                        acc[1] += ty;
                        acc[4] += tx * dx;
                        acc[5] += tx * dy;
                        acc[6] += ty * dy;
                    } else {
                        acc[4] += (T)0.5 * v_sigma * dx * dx;
                        acc[5] += v_sigma * dx * dy;
                        acc[6] += (T)0.5 * v_sigma * dy * dy;
                        const T gx = v_sigma * (g.a * dx + g.b * dy);
                        const T gy = v_sigma * (g.b * dx + g.c * dy);
                        acc[0] += gx;
                        acc[1] += gy;
                        acc[2] += M::abs_(gx);
                        acc[3] += M::abs_(gy);
                    }
                } else {
                    // csrc/gradient_aware_rasterizer.cu:201-315
                    const T dx = c.px - g.x;
                    const T dy = c.py - g.y;
                    const T sigma = sigma_ref<T>(g.a, g.b, g.c, dx, dy);
                    const T vis = M::exp_(-sigma);
                    const T alpha = M::min_(clamp, g.o * vis);
                    if (sigma < (T)0 || alpha < (T)1 / (T)255) continue;
                    touched = true;
                    const T sx = g.a * dx + g.b * dy;
                    const T sy = g.b * dx + g.c * dy;
                    const T a = g.a, b = g.b, cc = g.c;
                    const T ax = -alpha * sx;
                    const T ay = -alpha * sy;
                    const T axy = alpha * (sx * sy - b);
                    const T vo[3] = {c.vo0, c.vo1, c.vo2};
                    const T *vdx = c.vd, *vdy = c.vd + 3, *vdxy = c.vd + 6;
                    acc[7] += vo[0] * alpha + vdx[0] * ax + vdy[0] * ay + vdxy[0] * axy;
                    acc[8] += vo[1] * alpha + vdx[1] * ax + vdy[1] * ay + vdxy[1] * axy;
                    acc[9] += vo[2] * alpha + vdx[2] * ax + vdy[2] * ay + vdxy[2] * axy;
                    const T va = (vo[0] * g.r + vo[1] * g.g + vo[2] * g.bl) + c.vw;
                    const T vax = vdx[0] * g.r + vdx[1] * g.g + vdx[2] * g.bl;
                    const T vay = vdy[0] * g.r + vdy[1] * g.g + vdy[2] * g.bl;
                    const T vaxy = vdxy[0] * g.r + vdxy[1] * g.g + vdxy[2] * g.bl;
                    const T sx2 = sx * sx, sy2 = sy * sy, sxsy = sx * sy;
                    acc[0] += alpha * (va * sx + vax * (a - sx2) + vay * (b - sxsy) +
                                       vaxy * (sx2 * sy - (T)2 * b * sx - a * sy));
                    acc[1] += alpha * (va * sy + vax * (b - sxsy) + vay * (cc - sy2) +
                                       vaxy * (sx * sy2 - (T)2 * b * sy - cc * sx));
                    const T dx2 = dx * dx, dy2 = dy * dy, dxdy = dx * dy;
                    const T P = sxsy - b;
                    acc[4] += alpha * (va * (-(T)0.5 * dx2) + vax * ((T)0.5 * dx2 * sx - dx) +
                                       vay * ((T)0.5 * dx2 * sy) +
                                       vaxy * (-(T)0.5 * dx2 * P + dx * sy));
                    acc[5] += alpha * (va * (-dxdy) + vax * (dxdy * sx - dy) +
                                       vay * (dxdy * sy - dx) +
                                       vaxy * (-dxdy * P + dy * sy + dx * sx - (T)1));
                    acc[6] += alpha * (va * (-(T)0.5 * dy2) + vax * ((T)0.5 * dy2 * sx) +
                                       vay * ((T)0.5 * dy2 * sy - dy) +
                                       vaxy * (-(T)0.5 * dy2 * P + dy * sx));
                    acc[10] += vis * va;
                }
            }
            }
            for (int o = 1; o < (1 << lsplit); o <<= 1) {  // combine the lane group
#pragma unroll
                for (int q = 0; q < 11; ++q) {
                    if (LEAN && ((q == 10 && !GEN) || (!ABS && (q == 2 || q == 3)))) continue;
                    acc[q] += __shfl_xor_sync(FULL, acc[q], o);
                }
                touched = __shfl_xor_sync(FULL, (int)touched, o) || touched;
            }
            if (touched && part == 0) {
                if (LEAN && !GA && !direct) {
                    // v_xy = (a Sx + b Sy, b Sx + c Sy); v_conic = (Sxx/2, Sxy, Syy/2)
                    const T sx = acc[0], sy = acc[1];
                    const T a = kPairs ? (T)2 * g.a : g.a, c = kPairs ? (T)2 * g.c : g.c;
                    acc[0] = a * sx + g.b * sy;
                    acc[1] = g.b * sx + c * sy;
                    acc[4] *= (T)0.5;
                    acc[6] *= (T)0.5;
                }
                if (GA) {  // |sum over the reference warp| (= this region)
                    acc[2] = M::abs_(acc[0]);
                    acc[3] = M::abs_(acc[1]);
                }
                if constexpr (LEAN && ABS) {
                    // the general [N][12] layout
                    float4 *d4 = reinterpret_cast<float4 *>(packed + (size_t)s_ids[slot] * 12);
                    atomicAdd(d4, make_float4(acc[0], acc[1], acc[2], acc[3]));
                    atomicAdd(d4 + 1, make_float4(acc[4], acc[5], acc[6], acc[7]));
                    atomicAdd(d4 + 2, make_float4(acc[8], acc[9], GEN ? acc[10] : 0.f, 0.f));
                } else if constexpr (LEAN) {
                    // [xy, conic, rgb]
                    T *dst = packed + (size_t)s_ids[slot] * 8;
                    if constexpr (sizeof(T) == 4) {
                        float4 *d4 = reinterpret_cast<float4 *>(dst);
                        atomicAdd(d4, make_float4(acc[0], acc[1], acc[4], acc[5]));
                        atomicAdd(d4 + 1, make_float4(acc[6], acc[7], acc[8], acc[9]));
                    } else {
                        const T v[8] = {acc[0], acc[1], acc[4], acc[5],
                                        acc[6], acc[7], acc[8], acc[9]};
#pragma unroll
                        for (int q = 0; q < 8; ++q) atomicAdd(dst + q, v[q]);
                    }
                } else {
                    T *dst = packed + (size_t)s_ids[slot] * 12;
                    if constexpr (sizeof(T) == 4) {
                        float4 *d4 = reinterpret_cast<float4 *>(dst);
                        atomicAdd(d4, make_float4(acc[0], acc[1], acc[2], acc[3]));
                        atomicAdd(d4 + 1, make_float4(acc[4], acc[5], acc[6], acc[7]));
                        atomicAdd(d4 + 2, make_float4(acc[8], acc[9], acc[10], 0.f));
                    } else {
#pragma unroll
                        for (int q = 0; q < 11; ++q) atomicAdd(dst + q, acc[q]);
                    }
                }
            }
        }
    }
}

template <typename T, bool GA, bool LEAN, int MAXT, int MINB, bool ABS = false, int RR = 4,
          bool GEN = false>
__global__ void __launch_bounds__(MAXT, MINB)
raster_bwd_kernel(const BatchGeo geo, const int32_t *__restrict__ cum, int *work,
                  const int32_t *__restrict__ ids, const int2 *__restrict__ tile_bins,
                  const int32_t *__restrict__ d_total, const Rec<T> *__restrict__ recs,
                  const int32_t *__restrict__ final_idx, CotSrc<T> cot,
                  const T *__restrict__ v_dx, const T *__restrict__ v_dy,
                  const T *__restrict__ v_dxy, T clamp, T *__restrict__ packed) {
    __shared__ int s_end, s_slot;
    __shared__ __align__(8) unsigned long long s_mbar;
    const uint32_t bar = (uint32_t)__cvta_generic_to_shared(&s_mbar);
    uint32_t phase = 0;
    if (LIG_RASTER_BWD_BULK && LEAN && !GA && sizeof(T) == 4) {
        if (threadIdx.x == 0) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(1));
            asm volatile("fence.mbarrier_init.release.cluster;");
        }
        __syncthreads();
    }
    const int n_tiles = geo.total_tiles();
    for (int tile = next_tile(work, s_slot, true); tile < n_tiles;
         tile = next_tile(work, s_slot, false)) {
        const TileCtx tc = tile_ctx(geo, cum, d_total, tile);
        bwd_tile<T, GA, LEAN, ABS, RR, GEN>(tc, tile, ids, tile_bins, recs, final_idx, cot, v_dx,
                                            v_dy, v_dxy, clamp, packed, s_end, bar, phase);
    }
}

// ------------------------------------------------ gradient-aware backward
// Float, tiles of 16x16 (regions of 16x2 pixels) and 8x8 (8x4): the
// reference's warps, whose |sum| makes v_xy_abs.  As in the lean walk a lane
// takes one Gaussian (or 2 / 4 / 8 lanes share one) and loops over its
// region's pixels; columns c and c + W/2 of a row are evaluated as a pair in
// f32x2 arithmetic, and a pixel that fails the alpha test adds zeros.
//
// With d = pixel - mean, (sx, sy) = conic d, the four planes' cotangents
// V = (v, -v_dx, -v_dy, v_dxy) and, per colour channel,
//   E = V0 + V1 sx + V2 sy + V3 (sx sy - b),
// a pixel's term of the loss is alpha G, G = colour . E (+ v_wsum), so
//   v_colour = sum alpha E,
// and with gx = dG/dsx = V1.colour + V3.colour sy, gy likewise, the
// gradients of csrc/gradient_aware_rasterizer.cu:201-315 are linear in
//   S_ij = sum alpha G dx^i dy^j (i + j = 1, 2),  A = sum alpha gx,
//   B = sum alpha gy, A_x = sum alpha gx dx (A_y, B_x, B_y), D = sum alpha V3.colour:
//   v_xy    = conic (S10 - A, S01 - B)
//   v_conic = (A_x - S20/2, A_y + B_x - S11 - D, B_y - S02/2),
// applied once per Gaussian and region: 44 multiply-adds a pixel instead of
// the expanded formulas' 110.  dy is constant along a row, so the sums with dy
// come from row sums.
// Entries after a pixel's final index are not cut off: they fail the alpha
// test here exactly as they did in the forward.
// Bound by the FMA pipe (a packed operation takes two cycles of it; 62% busy at
// 61% of the issue slots) and the latency of its dependent chains (36% of the warps).  2047x1535 / 190k Gaussians: 518 us, against 1171
// for the scalar walk over the expanded formulas; 512^2 / 50k with opacities:
// 67 against 131.
struct alignas(16) GaPix {  // pixels (row, c) and (row, c + W/2)
    float v[12][2];         // plane-major: V0.rgb, V1.rgb, V2.rgb, V3.rgb
    float vw[2];
    float in[2];            // 1: inside the image (read by the skipping walk only)
};

// Pairs c0, c0 + CSTEP, ... (NCP of them) in two rows of a region (pix: the
// first row's entries, HW the entries per row), added to acc as [0, 1] v_xy, [4..6]
// v_conic, [7..9] v_rgb, [10] v_opacity.
template <int NCP, int CSTEP, int HW, bool OP, bool VW>
__device__ __forceinline__ void ga_rows(const Rec<float> &g, float clamp,
                                        const GaPix *__restrict__ pix, int c0, float px0,
                                        float py0, uint32_t cut, float (&acc)[11]) {
    const f2 AA = f2_dup(g.a), BB = f2_dup(g.b), CC = f2_dup(g.c), NB = f2_dup(-g.b);
    const f2 HALF = f2_dup(0.5f);
    const f2 CR = f2_dup(g.r), CG = f2_dup(g.g), CB = f2_dup(g.bl);
    const float hc = 0.5f * g.c;
    f2 wr[2], wx[2], wxx = f2_zero(), ar[2], br[2], ax = f2_zero(), bx = f2_zero();
    f2 dd = f2_zero(), cr = f2_zero(), cg = f2_zero(), cb = f2_zero();
    [[maybe_unused]] f2 vo = f2_zero();
    f2 DY[2], CDD[2];
    float dy[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        wr[r] = wx[r] = ar[r] = br[r] = f2_zero();
        dy[r] = (py0 + (float)r) - g.y;
        DY[r] = f2_dup(dy[r]);
        CDD[r] = f2_dup(__fmul_rn(__fmul_rn(hc, dy[r]), dy[r]));
    }
#pragma unroll
    for (int k = 0; k < NCP; ++k) {
        const int c = c0 + k * CSTEP;
        const f2 DX = f2_pack((px0 + (float)c) - g.x, (px0 + (float)(c + HW)) - g.x);
        const f2 AX = f2_mul(AA, DX), BX = f2_mul(BB, DX), HADX = f2_mul(HALF, AX);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const GaPix &e = pix[r * HW + c];
            const f2 S = f2_fma(BX, DY[r], f2_fma(HADX, DX, CDD[r]));
            float s0, s1;
            f2_unpack(S, s0, s1);
            const float vis0 = __expf(-s0), vis1 = __expf(-s1);
            const float al0 = fminf(clamp, OP ? g.o * vis0 : vis0);
            const float al1 = fminf(clamp, OP ? g.o * vis1 : vis1);
            bool no0, no1;
            if constexpr (!OP && LIG_RASTER_ALPHA_CUT) {
                no0 = __float_as_uint(s0) >= cut;
                no1 = __float_as_uint(s1) >= cut;
            } else {
                no0 = s0 < 0.f || al0 < 1.f / 255.f;
                no1 = s1 < 0.f || al1 < 1.f / 255.f;
            }
            const f2 AL = f2_pack(no0 ? 0.f : al0, no1 ? 0.f : al1);
            const f2 SX = f2_fma(BB, DY[r], AX), SY = f2_fma(CC, DY[r], BX);
            const f2 P = f2_fma(SX, SY, NB);
            f2 V[12];
#pragma unroll
            for (int q = 0; q < 6; ++q) {
                const ulonglong2 t = *reinterpret_cast<const ulonglong2 *>(e.v[2 * q]);
                V[2 * q] = f2{t.x};
                V[2 * q + 1] = f2{t.y};
            }
            const f2 ER = f2_fma(V[9], P, f2_fma(V[6], SY, f2_fma(V[3], SX, V[0])));
            const f2 EG = f2_fma(V[10], P, f2_fma(V[7], SY, f2_fma(V[4], SX, V[1])));
            const f2 EB = f2_fma(V[11], P, f2_fma(V[8], SY, f2_fma(V[5], SX, V[2])));
            cr = f2_fma(AL, ER, cr);
            cg = f2_fma(AL, EG, cg);
            cb = f2_fma(AL, EB, cb);
            f2 G = f2_fma(CB, EB, f2_fma(CG, EG, f2_mul(CR, ER)));
            const f2 VX = f2_fma(CB, V[5], f2_fma(CG, V[4], f2_mul(CR, V[3])));
            const f2 VY = f2_fma(CB, V[8], f2_fma(CG, V[7], f2_mul(CR, V[6])));
            const f2 VP = f2_fma(CB, V[11], f2_fma(CG, V[10], f2_mul(CR, V[9])));
            f2 W{0};
            if constexpr (VW) {
                W = f2{*reinterpret_cast<const unsigned long long *>(e.vw)};
                G = f2_add(G, W);
            }
            if constexpr (OP) {  // vis (v . colour + v_wsum), the reference's rule
                f2 VA = f2_fma(CB, V[2], f2_fma(CG, V[1], f2_mul(CR, V[0])));
                if constexpr (VW) VA = f2_add(VA, W);
                vo = f2_fma(f2_pack(no0 ? 0.f : vis0, no1 ? 0.f : vis1), VA, vo);
            }
            const f2 GX = f2_fma(VP, SY, VX), GY = f2_fma(VP, SX, VY);
            const f2 ALX = f2_mul(AL, DX);
            wr[r] = f2_fma(AL, G, wr[r]);
            wx[r] = f2_fma(ALX, G, wx[r]);
            wxx = f2_fma(f2_mul(ALX, DX), G, wxx);
            ar[r] = f2_fma(AL, GX, ar[r]);
            ax = f2_fma(ALX, GX, ax);
            br[r] = f2_fma(AL, GY, br[r]);
            bx = f2_fma(ALX, GY, bx);
            dd = f2_fma(AL, VP, dd);
        }
    }
    const float w0 = f2_sum(wr[0]), w1 = f2_sum(wr[1]), x0 = f2_sum(wx[0]), x1 = f2_sum(wx[1]);
    const float a0 = f2_sum(ar[0]), a1 = f2_sum(ar[1]), b0 = f2_sum(br[0]), b1 = f2_sum(br[1]);
    const float ux = x0 + x1 - (a0 + a1);                      // S10 - A
    const float wy0 = w0 * dy[0], wy1 = w1 * dy[1];
    const float uy = wy0 + wy1 - (b0 + b1);                    // S01 - B
    acc[0] += g.a * ux + g.b * uy;
    acc[1] += g.b * ux + g.c * uy;
    acc[4] += f2_sum(ax) - 0.5f * f2_sum(wxx);
    acc[5] += (a0 * dy[0] + a1 * dy[1]) + f2_sum(bx) - (x0 * dy[0] + x1 * dy[1]) - f2_sum(dd);
    acc[6] += (b0 * dy[0] + b1 * dy[1]) - 0.5f * (wy0 * dy[0] + wy1 * dy[1]);
    acc[7] += f2_sum(cr);
    acc[8] += f2_sum(cg);
    acc[9] += f2_sum(cb);
    if constexpr (OP) acc[10] += f2_sum(vo);
}

// One Gaussian over the region's pixels part, part + step, ... one at a time
// (rank = row W + column), skipping what fails the alpha test: records and
// tiles whose zeros could turn into NaN.  The expanded formulas of
// csrc/gradient_aware_rasterizer.cu:201-315.
template <int W>
__device__ __noinline__ void ga_pixels_skip(const Rec<float> &g, float clamp, const GaPix *pix,
                                            int part, int step, float px0, float py0, float *acc) {
    for (int j = part; j < 32; j += step) {
        const int row = j / W, col = j % W, h = col / (W / 2);
        const GaPix &e = pix[row * (W / 2) + col % (W / 2)];
        if (e.in[h] == 0.f) continue;
        const float dx = (px0 + (float)col) - g.x, dy = (py0 + (float)row) - g.y;
        const float sigma = sigma_ref<float>(g.a, g.b, g.c, dx, dy);
        const float vis = __expf(-sigma);
        const float alpha = fminf(clamp, g.o * vis);
        if (sigma < 0.f || alpha < 1.f / 255.f) continue;
        const float a = g.a, b = g.b, c = g.c;
        const float sx = a * dx + b * dy, sy = b * dx + c * dy;
        const float ax = -alpha * sx, ay = -alpha * sy, axy = alpha * (sx * sy - b);
        float vo[3], vx[3], vy[3], vp[3];
        for (int ch = 0; ch < 3; ++ch) {
            vo[ch] = e.v[ch][h];
            vx[ch] = -e.v[3 + ch][h];
            vy[ch] = -e.v[6 + ch][h];
            vp[ch] = e.v[9 + ch][h];
            acc[7 + ch] += vo[ch] * alpha + vx[ch] * ax + vy[ch] * ay + vp[ch] * axy;
        }
        const float va = (vo[0] * g.r + vo[1] * g.g + vo[2] * g.bl) + e.vw[h];
        const float vax = vx[0] * g.r + vx[1] * g.g + vx[2] * g.bl;
        const float vay = vy[0] * g.r + vy[1] * g.g + vy[2] * g.bl;
        const float vaxy = vp[0] * g.r + vp[1] * g.g + vp[2] * g.bl;
        const float sx2 = sx * sx, sy2 = sy * sy, sxsy = sx * sy;
        acc[0] += alpha * (va * sx + vax * (a - sx2) + vay * (b - sxsy) +
                           vaxy * (sx2 * sy - 2.f * b * sx - a * sy));
        acc[1] += alpha * (va * sy + vax * (b - sxsy) + vay * (c - sy2) +
                           vaxy * (sx * sy2 - 2.f * b * sy - c * sx));
        const float dx2 = dx * dx, dy2 = dy * dy, dxdy = dx * dy, P = sxsy - b;
        acc[4] += alpha * (va * (-0.5f * dx2) + vax * (0.5f * dx2 * sx - dx) +
                           vay * (0.5f * dx2 * sy) + vaxy * (-0.5f * dx2 * P + dx * sy));
        acc[5] += alpha * (va * (-dxdy) + vax * (dxdy * sx - dy) + vay * (dxdy * sy - dx) +
                           vaxy * (-dxdy * P + dy * sy + dx * sx - 1.f));
        acc[6] += alpha * (va * (-0.5f * dy2) + vax * (0.5f * dy2 * sx) +
                           vay * (0.5f * dy2 * sy - dy) + vaxy * (-0.5f * dy2 * P + dy * sx));
        acc[10] += vis * va;
    }
}

template <int W, bool OP, bool VW, int MINB>
__global__ void __launch_bounds__(W * W, MINB)
raster_bwd_ga_kernel(const BatchGeo geo, const int32_t *__restrict__ cum, int *work,
                     const int32_t *__restrict__ ids, const int2 *__restrict__ tile_bins,
                     const int32_t *__restrict__ d_total, const Rec<float> *__restrict__ recs,
                     const float *__restrict__ v_img, const float *__restrict__ v_wsum,
                     const float *__restrict__ v_dx, const float *__restrict__ v_dy,
                     const float *__restrict__ v_dxy, float clamp, float *__restrict__ packed) {
    constexpr int NT = W * W, HW = W / 2, NR = 32 / W;  // threads, pairs a row, rows a region
    constexpr int NW = NT / 32;
    __shared__ GaPix s_pix[NW * 16];
    __shared__ __align__(16) Rec<float> s_rec[NT];
    __shared__ int32_t s_ids[NT];
    __shared__ uint16_t s_list[NW][NT];
    __shared__ int s_slot;
    __shared__ __align__(8) unsigned long long s_mbar;
    const unsigned FULL = 0xffffffffu;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const uint32_t bar = (uint32_t)__cvta_generic_to_shared(&s_mbar);
    uint32_t phase = 0;
    if (tid == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(1));
        asm volatile("fence.mbarrier_init.release.cluster;");
    }
    __syncthreads();
    const int n_tiles = geo.total_tiles();
    const uint32_t cut = OP ? 0u : g_alpha_cut;
    const GaPix *my_pix = s_pix + w * 16;
    uint16_t *my_list = s_list[w];
    for (int tile = next_tile(work, s_slot, true); tile < n_tiles;
         tile = next_tile(work, s_slot, false)) {
        const TileCtx tc = tile_ctx(geo, cum, d_total, tile);
        if (tc.empty) continue;  // gradients stay zero (rasterize.py:156-161)
        const int2 range = tile_bins[tile];
        if (range.x >= range.y) continue;
        const Regions R = Regions::make(2, W);
        bulk_records(bar, s_rec, s_ids, ids, recs, range.x, min(NT, range.y - range.x));
        // stage this thread's pixel: rank tid of the tile
        const int col = tid % W, gx = tc.tx0 + col, gy = tc.ty0 + tid / W;
        const bool inside = gx < tc.W && gy < tc.H;
        const int p = inside ? tc.poff + gy * tc.W + gx : 0;
        float v[13];
#pragma unroll
        for (int ch = 0; ch < 3; ++ch) {
            v[ch] = inside ? v_img[3 * p + ch] : 0.f;
            v[3 + ch] = inside ? -v_dx[3 * p + ch] : 0.f;
            v[6 + ch] = inside ? -v_dy[3 * p + ch] : 0.f;
            v[9 + ch] = inside ? v_dxy[3 * p + ch] : 0.f;
        }
        v[12] = VW && inside ? v_wsum[p] : 0.f;
        GaPix &mine = s_pix[w * 16 + (lane / W) * HW + col % HW];
        bool tame_cot = true;
        mine.in[col / HW] = inside ? 1.f : 0.f;
#pragma unroll
        for (int q = 0; q < 13; ++q) {
            tame_cot = tame_cot && fabsf(v[q]) < kTameCot;
            if (q < 12) mine.v[q][col / HW] = v[q];
            else mine.vw[col / HW] = v[q];
        }
        const bool wild = __syncthreads_or(!tame_cot);
        const float px0 = (float)tc.tx0 + 0.5f, py0 = (float)(tc.ty0 + w * NR) + 0.5f;
        for (int base = range.x; base < range.y; base += NT) {
            const int cnt = min(NT, range.y - base);
            if (base != range.x) {  // everyone is done with the previous batch
                __syncthreads();
                bulk_records(bar, s_rec, s_ids, ids, recs, base, cnt);
            }
            const bool ok = mbar_wait(bar, phase);
            phase ^= 1u;
            // as in bwd_tile: a wait that gave up abandons the tile
            if (__syncthreads_or(!ok)) {
                if (tid == 0) atomicAdd(&g_wait_timeouts, 1u);
                (void)mbar_wait(bar, phase ^ 1u);
                break;
            }
            // the batch's Gaussians that reach this region, in list order
            int nmine = 0;
            for (int m = 0; m * 32 < cnt; ++m) {
                const int t = m * 32 + lane;
                const bool hit =
                    t < cnt && region_hit<float, true, false>(s_rec[t], R, w, tc.tx0, tc.ty0);
                const uint32_t mask = __ballot_sync(FULL, hit);
                if (hit) my_list[nmine + __popc(mask & ((1u << lane) - 1u))] = (uint16_t)t;
                nmine += __popc(mask);
            }
            __syncwarp();
            for (int g0 = 0, lsplit = 0; g0 < nmine; g0 += 32 >> lsplit) {
                const int left = min(32, nmine - g0);
                lsplit = left <= LIG_RASTER_GA_BWD_SPLIT3   ? 3
                         : left <= LIG_RASTER_GA_BWD_SPLIT2 ? 2
                         : left <= LIG_RASTER_GA_BWD_SPLIT1 ? 1 : 0;
                const int gi = lane >> lsplit, part = lane & ((1 << lsplit) - 1);
                const bool act = gi < left;
                const int slot = act ? (int)my_list[g0 + gi] : 0;
                const Rec<float> g = s_rec[slot];
                float acc[11];
#pragma unroll
                for (int q = 0; q < 11; ++q) acc[q] = 0.f;
                if (act && (wild || !(g.wx >= 0.f))) {
                    float t[11] = {};
                    ga_pixels_skip<W>(s_rec[slot], clamp, my_pix, part, 1 << lsplit, px0, py0, t);
#pragma unroll
                    for (int q = 0; q < 11; ++q) acc[q] = t[q];
                } else if (act) {
                    // row pairs: one for W = 16, two for W = 8 (8 lanes: one each)
                    const int rb = W == 8 && lsplit == 3 ? part >> 2 : 0;
                    const int re = W == 8 && lsplit == 3 ? rb + 1 : NR / 2;
#pragma unroll 1
                    for (int rp = rb; rp < re; ++rp) {
                        const GaPix *rows = my_pix + 2 * rp * HW;
                        const float py = py0 + (float)(2 * rp);
                        switch (lsplit) {
                        case 0:
                            ga_rows<HW, 1, HW, OP, VW>(g, clamp, rows, 0, px0, py, cut, acc);
                            break;
                        case 1:
                            ga_rows<HW / 2, 2, HW, OP, VW>(g, clamp, rows, part, px0, py, cut, acc);
                            break;
                        case 2:
                            ga_rows<HW / 4, 4, HW, OP, VW>(g, clamp, rows, part, px0, py, cut, acc);
                            break;
                        default:
                            ga_rows<1, 8, HW, OP, VW>(g, clamp, rows, part & (HW - 1), px0, py, cut,
                                                      acc);
                            break;
                        }
                    }
                }
                for (int o = 1; o < (1 << lsplit); o <<= 1) {  // combine the lane group
#pragma unroll
                    for (int q = 0; q < 11; ++q) {
                        if (q == 2 || q == 3 || (!OP && q == 10)) continue;
                        acc[q] += __shfl_xor_sync(FULL, acc[q], o);
                    }
                }
                if (act && part == 0) {
                    // v_xy_abs: |sum over the reference's warp| (= this region)
                    float4 *d4 = reinterpret_cast<float4 *>(packed + (size_t)s_ids[slot] * 12);
                    atomicAdd(d4, make_float4(acc[0], acc[1], fabsf(acc[0]), fabsf(acc[1])));
                    atomicAdd(d4 + 1, make_float4(acc[4], acc[5], acc[6], acc[7]));
                    atomicAdd(d4 + 2, make_float4(acc[8], acc[9], OP ? acc[10] : 0.f, 0.f));
                }
            }
        }
    }
}

// Packed per-Gaussian gradients [N][12] -> the five output arrays of the ABI.
template <typename T>
__global__ void unpack_lean_grads_kernel(int n, const T *__restrict__ packed, Grads<T> out) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const T *g = packed + (size_t)i * 8;
    out.v_xy[2 * i] = g[0];
    out.v_xy[2 * i + 1] = g[1];
    out.v_abs[2 * i] = 0;
    out.v_abs[2 * i + 1] = 0;
    out.v_conic[3 * i] = g[2];
    out.v_conic[3 * i + 1] = g[3];
    out.v_conic[3 * i + 2] = g[4];
    out.v_rgb[3 * i] = g[5];
    out.v_rgb[3 * i + 1] = g[6];
    out.v_rgb[3 * i + 2] = g[7];
}

template <typename T>
__global__ void unpack_grads_kernel(int n, const T *__restrict__ packed, Grads<T> out) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const T *g = packed + (size_t)i * 12;
    out.v_xy[2 * i] = g[0];
    out.v_xy[2 * i + 1] = g[1];
    out.v_abs[2 * i] = g[2];
    out.v_abs[2 * i + 1] = g[3];
    out.v_conic[3 * i] = g[4];
    out.v_conic[3 * i + 1] = g[5];
    out.v_conic[3 * i + 2] = g[6];
    out.v_rgb[3 * i] = g[7];
    out.v_rgb[3 * i + 1] = g[8];
    out.v_rgb[3 * i + 2] = g[9];
    if (out.v_opac) out.v_opac[i] = g[10];
}

// ------------------------------------------------------------------ host
template <typename T>
int pack(int n, const void *xys, const void *con, const void *col, const void *op, void *ws,
         size_t ws_bytes, cudaStream_t s, bool half = false, T *zero = nullptr,
         int zero_stride = 0, bool tame = false, uint32_t *ticket = nullptr) {
    if (ws_bytes < sizeof(Rec<T>) * (size_t)n) return LIG_ERR_WORKSPACE;
    if ((reinterpret_cast<uintptr_t>(ws) & 15) != 0) return LIG_ERR_INVALID;  // 16-byte records
    if (n > 0) {
        auto k = half ? (tame ? pack_kernel<T, true, true> : pack_kernel<T, true>)
                      : (tame ? pack_kernel<T, false, true> : pack_kernel<T, false>);
        k<<<(n + 255) / 256, 256, 0, s>>>(n, (const T *)xys, (const T *)con, (const T *)col,
                                          (const T *)op, (Rec<T> *)ws, zero, zero_stride, ticket);
    } else if (ticket) {
        cudaMemsetAsync(ticket, 0, sizeof(*ticket), s);
    }
    note_launches(n > 0 ? 1 : 0);
    LIG_LAUNCH_CHECK();
    return LIG_OK;
}

// Opt a kernel into `bytes` of dynamic shared memory, once per (kernel,
// device, size): repeated calls cost nothing, and none is made during a
// stream capture after the first eager call.
#ifndef LIG_RASTER_CARVEOUT
#define LIG_RASTER_CARVEOUT -1  // shared-memory carveout percent; -1: driver default
#endif

// Opts a kernel into its dynamic shared memory, once per device and size.  A
// launch is given 48 KB unasked, its static shared memory included: a kernel
// that comes within kStaticSmem of that asks too.
constexpr size_t kDefaultSmem = 48 * 1024, kStaticSmem = 4 * 1024;
inline bool set_dyn_smem(const void *fn, size_t bytes) {
    const bool ask = bytes > kDefaultSmem - kStaticSmem;
    if (!ask && LIG_RASTER_CARVEOUT < 0) return true;
    static std::mutex mu;
    static std::vector<std::tuple<const void *, int, size_t>> done;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return false;
    std::lock_guard<std::mutex> lock(mu);
    for (auto &e : done)
        if (std::get<0>(e) == fn && std::get<1>(e) == dev && std::get<2>(e) >= bytes) return true;
    if (ask &&
        cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes) !=
            cudaSuccess)
        return false;
    if (LIG_RASTER_CARVEOUT >= 0 &&
        cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout,
                             LIG_RASTER_CARVEOUT) != cudaSuccess)
        return false;
    done.emplace_back(fn, dev, bytes);
    return true;
}

// Grid of a persistent launch: every CTA that fits on the device at once.
inline int persistent_grid(const void *fn, int threads, size_t smem) {
    static std::mutex mu;
    static std::vector<std::tuple<const void *, int, int, size_t, int>> cache;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    std::lock_guard<std::mutex> lock(mu);
    for (auto &e : cache)
        if (std::get<0>(e) == fn && std::get<1>(e) == dev && std::get<2>(e) == threads &&
            std::get<3>(e) == smem)
            return std::get<4>(e);
    int per_sm = 0, sms = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, threads, smem) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return 0;
    const int g = per_sm * sms;
    cache.emplace_back(fn, dev, threads, smem, g);
    return g;
}

// How a raster kernel walks the flattened (image, tile) list.
struct TileWalk {
    const int32_t *cum = nullptr;  // per-image empty test (batched); null: *d_total
    int *work = nullptr;           // persistent: global work counter; null: CTA per tile
};

// Loss outputs of the fused-L2 forward (with a target).
template <typename T> struct L2Out {
    T *loss = nullptr, *per_image = nullptr;
};

inline int raster_fwd_ga(const BatchGeo &geo, TileWalk walk, const int32_t *ids,
                         const int32_t *bins, const int32_t *d_total, const void *ws, bool op,
                         float *img, float *wsum, float *dx, float *dy, float *dxy, int32_t *fin,
                         cudaStream_t s) {
    const int nt = 32 * Regions::make(1, geo.B).count;  // at most 128; 512 for B > 16
    const size_t sm = (size_t)nt * sizeof(Rec<float>);
    auto fn = geo.B > 16 ? (op ? raster_fwd_ga_kernel<true, 512, 1> : raster_fwd_ga_kernel<false, 512, 1>)
              : op       ? raster_fwd_ga_kernel<true, 128, LIG_RASTER_GA_MINB>
                         : raster_fwd_ga_kernel<false, 128, LIG_RASTER_GA_MINB>;
    int grid = geo.total_tiles();
    if (walk.work) {
        const int pg = persistent_grid((const void *)fn, nt, sm);
        if (pg <= 0) return launch_refused();
        grid = grid < pg ? grid : pg;
        cudaMemsetAsync(walk.work, 0, sizeof(int), s);
    }
    fn<<<grid, nt, sm, s>>>(geo, walk.cum, walk.work, ids, (const int2 *)bins, d_total,
                            (const Rec<float> *)ws, img, wsum, dx, dy, dxy, fin);
    note_launches(1);
    LIG_LAUNCH_CHECK();
    return LIG_OK;
}

template <typename T>
int raster_fwd(const BatchGeo &geo, TileWalk walk, const int32_t *ids, const int32_t *bins,
               const int32_t *d_total, const void *xys, const void *con, const void *col,
               const void *op, void *ws, size_t ws_bytes, void *img, void *wsum, void *dx,
               void *dy, void *dxy, int32_t *fin, cudaStream_t s,
               L2Fwd<T> l2 = L2Fwd<T>{nullptr, nullptr}, L2Out<T> l2o = L2Out<T>{},
               bool have_recs = false, AdamPro pro = AdamPro{}) {
    const int n = geo.total_points();
    const bool ga = dx != nullptr;
    const bool fused = l2.target || l2.target_u8;
    // the sum forward reads the halved conic (see sigma_half)
    // (have_recs: the fit step's fit_project_kernel has written the records and
    // cleared the ticket)
    double *chunk_sum = l2.tile_partial + geo.total_tiles();
    uint32_t *ticket = fused ? loss_ticket(l2.tile_partial, geo.total_tiles()) : nullptr;
    if (!have_recs) {
        const int rc = pack<T>(n, xys, con, col, op, ws, ws_bytes, s, !ga, nullptr, 0, ga, ticket);
        if (rc) return rc;
    }
    // float, gradient-aware: the pair walk on 8x8 regions, but for tiles that fill
    // those by a half or two thirds where 8x4 regions hold twice or a fifth more
    // (one pixel a lane / pairs: 4x4 tiles, 512^2 / 20k 36 / 43 us, 20x20 35 / 37)
    if constexpr (sizeof(T) == 4) {
        if (ga && !(geo.B <= 4 || (geo.B > 16 && geo.B <= 20)))
            return raster_fwd_ga(geo, walk, ids, bins, d_total, ws, op != nullptr, (float *)img,
                                 (float *)wsum, (float *)dx, (float *)dy, (float *)dxy, fin, s);
    }
    // (tiles of up to 8 rows would leave half of an 8x16 region outside: 8x8
    // tiles at 2048^2 / 150k take 126 us with two pixels a lane, 190 with four)
    const bool ppl4 = !ga && geo.B > 8 && geo.total_tiles() >= LIG_RASTER_PPL4_MIN_TILES;
    const int nt = 32 * Regions::make(ga ? 0 : (ppl4 ? 3 : 1), geo.B).count;
    const size_t sm = (size_t)nt * sizeof(Rec<T>);
    using K = void (*)(const BatchGeo, const int32_t *, int *, const int32_t *, const int2 *,
                       const int32_t *, const Rec<T> *, T *, T *, T *, T *, T *, int32_t *,
                       L2Fwd<T>);
    const bool small = nt <= 256;
    constexpr int FM = LIG_RASTER_FWD_MINB;
    auto sum = [&](auto ppl, auto op_t, auto fin_t, auto ws_t) -> K {
        constexpr int P = decltype(ppl)::value;
        constexpr bool O = decltype(op_t)::value, F = decltype(fin_t)::value,
                       S = decltype(ws_t)::value;
        // tiles of up to 16x16: at most 64 threads with four pixels a lane, 128 with two
        constexpr int kMaxT = P == 4 ? 64 : 128;
        // resident CTAs per SM: the fused loss's 8192^2 / 2M 1378 us with 16 (64
        // registers), 1436 with 14; with weight sums and indices eight views
        // 401 with 14, 412 with 16 (spilling); 8x8 regions, 512^2 / 50k 26.8
        // with 9, 27.8 with 8, 27.4 with 10 (767x1023 with opacities 63 / 65 / 69)
        // (double: 6; 512^2 / 20k 48.6 us with 6, 49.4 with 8, 51.6 with 9)
        constexpr int kMinB = P == 4 ? (S ? 14 : 16) : sizeof(T) == 8 ? 6 : 9;
        return nt <= kMaxT ? raster_fwd_kernel<T, false, P, kMaxT, kMinB, O, F, S>
                           : raster_fwd_kernel<T, false, P, 512, 2, O, F, S>;
    };
    auto pick = [&](auto ppl) -> K {
        using std::false_type;
        using std::true_type;
        // (double takes the walk with opacities, 1 where there are none: 512^2 / 20k
        // 45.7 us, 48.6 without the product)
        if (!fused)
            return op || sizeof(T) == 8 ? sum(ppl, true_type{}, true_type{}, true_type{})
                                        : sum(ppl, false_type{}, true_type{}, true_type{});
        return op    ? sum(ppl, true_type{}, true_type{}, false_type{})
               : fin ? sum(ppl, false_type{}, true_type{}, false_type{})
                     : sum(ppl, false_type{}, false_type{}, false_type{});
    };
    K fn;
    if (ga) {
        fn = small ? raster_fwd_kernel<T, true, 1, 256, FM> : raster_fwd_kernel<T, true, 1, 1024, 1>;
    } else {
        fn = ppl4 ? pick(std::integral_constant<int, 4>{}) : pick(std::integral_constant<int, 2>{});
    }
    if (!set_dyn_smem((const void *)fn, sm)) return launch_refused();
    int grid = geo.total_tiles();
    if (walk.work) {
        const int pg = persistent_grid((const void *)fn, nt, sm);
        if (pg <= 0) return launch_refused();
        grid = grid < pg ? grid : pg;
        cudaMemsetAsync(walk.work, 0, sizeof(int), s);
    }
    fn<<<grid, nt, sm, s>>>(geo, walk.cum, walk.work, ids, (const int2 *)bins, d_total,
                            (const Rec<T> *)ws, (T *)img, (T *)wsum, ga ? (T *)dx : nullptr,
                            ga ? (T *)dy : nullptr, ga ? (T *)dxy : nullptr, fin, l2);
    int launches = 1;
    if (fused) {
        const TileChunks ch = tile_chunks(geo);
        l2_loss_kernel<T><<<ch.chunk_off[geo.n_img] + (pro.out ? 1 : 0), 256, 0, s>>>(
            geo, ch, l2.tile_partial, chunk_sum, ticket, l2o.loss, l2o.per_image, pro);
        ++launches;
    }
    note_launches(launches);
    LIG_LAUNCH_CHECK();
    return LIG_OK;
}

inline int raster_bwd_ga(const BatchGeo &geo, TileWalk walk, const int32_t *ids,
                         const int32_t *bins, const int32_t *d_total, const void *ws, bool op,
                         const CotSrc<float> &cot, const float *v_dx, const float *v_dy,
                         const float *v_dxy, float clamp, float *packed, cudaStream_t s) {
    constexpr int M = LIG_RASTER_GA_BWD_MINB;
    const bool vw = cot.v_wsum != nullptr;
    auto fn = geo.B == 16 ? (op ? (vw ? raster_bwd_ga_kernel<16, true, true, M>
                                      : raster_bwd_ga_kernel<16, true, false, M>)
                                : (vw ? raster_bwd_ga_kernel<16, false, true, M>
                                      : raster_bwd_ga_kernel<16, false, false, M>))
                          : (op ? (vw ? raster_bwd_ga_kernel<8, true, true, 4 * M>
                                      : raster_bwd_ga_kernel<8, true, false, 4 * M>)
                                : (vw ? raster_bwd_ga_kernel<8, false, true, 4 * M>
                                      : raster_bwd_ga_kernel<8, false, false, 4 * M>));
    const int nt = geo.B * geo.B;
    int grid = geo.total_tiles();
    if (walk.work) {
        const int pg = persistent_grid((const void *)fn, nt, 0);
        if (pg <= 0) return launch_refused();
        grid = grid < pg ? grid : pg;
        cudaMemsetAsync(walk.work, 0, sizeof(int), s);
    }
    fn<<<grid, nt, 0, s>>>(geo, walk.cum, walk.work, ids, (const int2 *)bins, d_total,
                           (const Rec<float> *)ws, cot.v_img, cot.v_wsum, v_dx, v_dy, v_dxy, clamp,
                           packed);
    return LIG_OK;
}

// Backward workspace: packed records [N] followed by packed gradients [N][12].
template <typename T>
inline size_t bwd_grad_offset(int n) {
    return (sizeof(Rec<T>) * (size_t)(n > 0 ? n : 1) + 255) & ~(size_t)255;
}

template <typename T>
int raster_bwd(const BatchGeo &geo, TileWalk walk, const int32_t *ids, const int32_t *bins,
               const int32_t *d_total, const void *xys, const void *con, const void *col,
               const void *op, const int32_t *fin, CotSrc<T> cot, const void *v_dx,
               const void *v_dy, const void *v_dxy, double clamp, void *ws, size_t ws_bytes,
               void *v_xy, void *v_abs, void *v_con, void *v_rgb, void *v_op, cudaStream_t s,
               bool prepacked = false) {
    const int n = geo.total_points();
    const size_t goff = bwd_grad_offset<T>(n);
    if (ws_bytes < goff + sizeof(T) * 12 * (size_t)n) return LIG_ERR_WORKSPACE;
    const bool ga = v_dx != nullptr;
    // the fused-loss backward without opacities needs neither |v_xy| nor an
    // opacity gradient (nor a wsum cotangent)
    const bool lean = !ga && !cot.v_img && !cot.v_wsum && !op && !v_op;
    // an explicit image cotangent without wsum cotangent or opacities (the
    // drop-in API under autograd, LIG's own training loop): the same lean
    // walk plus the per-pixel |v_xy| sums the reference returns (float)
    const bool lean_abs = !ga && cot.v_img && !cot.v_wsum && !op && !v_op &&
                          sizeof(T) == 4 && LIG_RASTER_BWD_F2;
    const int stride = lean ? 8 : 12;
    T *packed = reinterpret_cast<T *>((char *)ws + goff);
    // float gradient-aware: 16x16 and 8x8 tiles, whose reference warps are
    // blocks of pixels
    const bool ga_pairs = ga && sizeof(T) == 4 && cot.v_img && (geo.B == 16 || geo.B == 8);
    // float sum backward with opacities or a wsum cotangent: the pair walk too, but for
    // 2x2 tiles, which fill an eighth of its 8x4 regions (300x333 / 8k: 49 us a call,
    // 46 with the scalar walk, which skips the pixels outside; 3x3 33, 38 scalar)
    const bool general = !ga && !lean && !lean_abs;
    const bool gen = general && sizeof(T) == 4 && geo.B > 2;
    // records (halved conic for the pair walks), and the packed gradients cleared
    // in the same pass; prepacked (lean): the forward left both in ws, and the
    // gradients stay packed
    int rc = LIG_OK;
    if (!prepacked)
        rc = pack<T>(n, xys, con, col, op, ws, goff, s,
                     sizeof(T) == 4 && (lean || lean_abs || gen), packed, stride, ga_pairs || gen);
    if (rc) return rc;
    const T cl = (T)(clamp > 0 ? clamp : (ga ? 0.999 : 0.99));
    Grads<T> g{(T *)v_xy, (T *)v_abs, (T *)v_con, (T *)v_rgb, (T *)v_op};
    auto unpack = [&]() {
        if (n > 0 && lean) unpack_lean_grads_kernel<T><<<(n + 255) / 256, 256, 0, s>>>(n, packed, g);
        else if (n > 0) unpack_grads_kernel<T><<<(n + 255) / 256, 256, 0, s>>>(n, packed, g);
        note_launches(n > 0 ? 1 : 0);
    };
    // min(clamp, exp(-sigma)) < 1/255 at every pixel: the cleared sums are the
    // gradients (the walks' alpha cut stands for the rule from 1/255 on)
    if (!prepacked && cl < (T)1 / (T)255) {
        unpack();
        LIG_LAUNCH_CHECK();
        return LIG_OK;
    }
    if constexpr (sizeof(T) == 4) {
        if (ga_pairs) {
            rc = raster_bwd_ga(geo, walk, ids, bins, d_total, ws, op || v_op, cot, (const T *)v_dx,
                               (const T *)v_dy, (const T *)v_dxy, cl, packed, s);
            if (rc) return rc;
            note_launches(1);
            unpack();
            LIG_LAUNCH_CHECK();
            return LIG_OK;
        }
    }
    const bool large = geo.total_tiles() >= LIG_RASTER_BWD_LARGE_MIN_TILES;
    // the float pair walks of large images: taller regions (tiles up to 16x16)
    const double density = (double)n / (double)geo.total_pixels();
    // (8x8 tiles fill half of an 8x16 region: 2048^2 / 150k 185 us with 8x8
    // regions, 275 with 8x16)
    const int rr_auto = density <= LIG_RASTER_BWD_R16_MAX_DENSITY && geo.B > 8 ? 16 : 8;
    // (tiles of up to 4 rows fill a quarter of an 8x8 region: general walk, 4x4 tiles at
    // 512^2 / 20k 45 us with 8x4 regions, 66 with 8x8)
    const int rr = (LIG_RASTER_BWD_RROWS != 4 && sizeof(T) == 4 && LIG_RASTER_BWD_F2 &&
                    !ga && large && geo.B <= 16 && !(general && geo.B <= 4))
                       ? (LIG_RASTER_BWD_RROWS ? LIG_RASTER_BWD_RROWS : rr_auto)
                       : 4;
    const int nt = 32 * Regions::make(ga ? 2 : (rr == 8 ? 1 : rr == 16 ? 3 : 0), geo.B).count;
    const int nw = nt / 32;
    const size_t pix = ga ? sizeof(PixRec<T, true>) : sizeof(PixRec<T, false>) * (rr == 16 ? 2 : 1);
    const size_t sm = (size_t)nt * pix + (size_t)nt * (sizeof(Rec<T>) + 2 * sizeof(uint32_t)) +
                      (size_t)nw * nt * sizeof(uint16_t);
    using K = void (*)(const BatchGeo, const int32_t *, int *, const int32_t *, const int2 *,
                       const int32_t *, const Rec<T> *, const int32_t *, CotSrc<T>, const T *,
                       const T *, const T *, T, T *);
    const bool small = nt <= 256;
    constexpr bool kAbs = sizeof(T) == 4 && LIG_RASTER_BWD_F2;
    constexpr int kMin = LIG_RASTER_BWD_LEAN_MINB, kMinL = LIG_RASTER_BWD_LEAN_MINB_LARGE;
    K fn;
    if (ga) {
        fn = small ? raster_bwd_kernel<T, true, false, 256, LIG_RASTER_BWD_MINB>
                   : raster_bwd_kernel<T, true, false, 1024, 1>;
    } else if (lean) {
        fn = !small  ? raster_bwd_kernel<T, false, true, 1024, 1>
             : large ? raster_bwd_kernel<T, false, true, 256, kMinL>
                     : raster_bwd_kernel<T, false, true, 256, kMin>;
    } else if constexpr (kAbs) {
        if (lean_abs)
            fn = !small  ? raster_bwd_kernel<T, false, true, 1024, 1, true>
                 : large ? raster_bwd_kernel<T, false, true, 256, kMinL, true>
                         : raster_bwd_kernel<T, false, true, 256, kMin, true>;
        else if (!gen)
            fn = raster_bwd_kernel<T, false, false, 256, LIG_RASTER_BWD_MINB>;
        else
            fn = !small  ? raster_bwd_kernel<T, false, true, 1024, 1, true, 4, true>
                         : raster_bwd_kernel<T, false, true, 256, LIG_RASTER_GEN_MINB, true, 4, true>;
    } else {
        fn = small ? raster_bwd_kernel<T, false, false, 256, LIG_RASTER_BWD_MINB>
                   : raster_bwd_kernel<T, false, false, 1024, 1>;
    }
    if constexpr (kAbs) {
        constexpr int M8 = LIG_RASTER_BWD_RROWS_MINB, M16 = LIG_RASTER_BWD_R16_MINB;
        if (rr == 8)
            fn = gen        ? raster_bwd_kernel<T, false, true, 128, LIG_RASTER_GEN_R8_MINB, true, 8, true>
                 : lean_abs ? raster_bwd_kernel<T, false, true, 128, M8, true, 8>
                            : raster_bwd_kernel<T, false, true, 128, M8, false, 8>;
        else if (rr == 16)
            fn = gen        ? raster_bwd_kernel<T, false, true, 64, LIG_RASTER_GEN_R16_MINB, true, 16, true>
                 : lean_abs ? raster_bwd_kernel<T, false, true, 64, M16, true, 16>
                            : raster_bwd_kernel<T, false, true, 64, M16, false, 16>;
    }
    if (!set_dyn_smem((const void *)fn, sm)) return launch_refused();
    int grid = geo.total_tiles();
    if (walk.work) {
        const int pg = persistent_grid((const void *)fn, nt, sm);
        if (pg <= 0) return launch_refused();
        grid = grid < pg ? grid : pg;
        cudaMemsetAsync(walk.work, 0, sizeof(int), s);
    }
    fn<<<grid, nt, sm, s>>>(geo, walk.cum, walk.work, ids, (const int2 *)bins, d_total,
                            (const Rec<T> *)ws, fin, cot, ga ? (const T *)v_dx : nullptr,
                            ga ? (const T *)v_dy : nullptr, ga ? (const T *)v_dxy : nullptr, cl,
                            packed);
    note_launches(1);
    if (!prepacked) unpack();
    LIG_LAUNCH_CHECK();
    return LIG_OK;
}

inline bool raster_args_ok(int H, int W, int B, int n) {
    // pixel-channel indices are 32-bit
    return H > 0 && W > 0 && B >= 2 && B <= 32 && n >= 0 &&
           3ll * H * W <= 0x7fffffffll;
}

}  // namespace lig

using namespace lig;

extern "C" size_t lig_raster_workspace_bytes(int dtype, int n) {
    size_t m = (size_t)(n > 0 ? n : 1);
    if (dtype == LIG_F64) return bwd_grad_offset<double>(n) + sizeof(double) * 12 * m;
    return bwd_grad_offset<float>(n) + sizeof(float) * 12 * m;
}

extern "C" int lig_raster_fwd(int dtype, int H, int W, int B, int n, const int32_t *ids,
                              const int32_t *bins, const int32_t *d_total, const void *xys,
                              const void *con, const void *col, const void *op, void *ws,
                              size_t ws_bytes, void *img, void *wsum, void *dx, void *dy,
                              void *dxy, int32_t *fin, void *stream) {
    if (!raster_args_ok(H, W, B, n) || !bins || !d_total || !img || !wsum || !fin || !ws ||
        (n > 0 && (!xys || !con || !col)) || ((dx || dy || dxy) && !(dx && dy && dxy)))
        return LIG_ERR_INVALID;
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype == LIG_F32)
        return raster_fwd<float>(BatchGeo::single(H, W, B, n), TileWalk{}, ids, bins, d_total,
                                 xys, con, col, op, ws, ws_bytes, img, wsum, dx, dy, dxy, fin, s);
    if (dtype == LIG_F64)
        return raster_fwd<double>(BatchGeo::single(H, W, B, n), TileWalk{}, ids, bins, d_total,
                                  xys, con, col, op, ws, ws_bytes, img, wsum, dx, dy, dxy, fin, s);
    return LIG_ERR_INVALID;
}

extern "C" int lig_raster_bwd(int dtype, int H, int W, int B, int n, const int32_t *ids,
                              const int32_t *bins, const int32_t *d_total, const void *xys,
                              const void *con, const void *col, const void *op,
                              const int32_t *fin, const void *v_img, const void *v_wsum,
                              const void *v_dx, const void *v_dy, const void *v_dxy,
                              double clamp, void *ws, size_t ws_bytes, void *v_xy, void *v_abs,
                              void *v_con, void *v_rgb, void *v_op, void *stream) {
    if (!raster_args_ok(H, W, B, n) || !bins || !d_total || !fin || !v_img || !ws ||
        (n > 0 && (!xys || !con || !col || !v_xy || !v_abs || !v_con || !v_rgb)) ||
        ((v_dx || v_dy || v_dxy) && !(v_dx && v_dy && v_dxy)))
        return LIG_ERR_INVALID;
    cudaStream_t s = (cudaStream_t)stream;
    if (n == 0) return LIG_OK;
    if (dtype == LIG_F32) {
        CotSrc<float> cot{(const float *)v_img, (const float *)v_wsum, nullptr, nullptr, nullptr, 0.f};
        return raster_bwd<float>(BatchGeo::single(H, W, B, n), TileWalk{}, ids, bins, d_total,
                                 xys, con, col, op, fin, cot,
                                 v_dx, v_dy, v_dxy, clamp, ws, ws_bytes, v_xy, v_abs, v_con,
                                 v_rgb, v_op, s);
    }
    if (dtype == LIG_F64) {
        CotSrc<double> cot{(const double *)v_img, (const double *)v_wsum, nullptr, nullptr, nullptr, 0.0};
        return raster_bwd<double>(BatchGeo::single(H, W, B, n), TileWalk{}, ids, bins, d_total,
                                  xys, con, col, op, fin, cot,
                                  v_dx, v_dy, v_dxy, clamp, ws, ws_bytes, v_xy, v_abs, v_con,
                                  v_rgb, v_op, s);
    }
    return LIG_ERR_INVALID;
}

extern "C" int lig_raster_bwd_l2(int dtype, int H, int W, int B, int n, const int32_t *ids,
                                 const int32_t *bins, const int32_t *d_total, const void *xys,
                                 const void *con, const void *col, const void *op,
                                 const int32_t *fin, const void *img, const void *target,
                                 const void *grad_loss, double clamp, void *ws, size_t ws_bytes,
                                 void *v_xy, void *v_abs, void *v_con, void *v_rgb, void *v_op,
                                 void *stream) {
    if (!raster_args_ok(H, W, B, n) || !bins || !d_total || !fin || !img || !target ||
        !grad_loss || !ws || (n > 0 && (!xys || !con || !col || !v_xy || !v_abs || !v_con || !v_rgb)))
        return LIG_ERR_INVALID;
    cudaStream_t s = (cudaStream_t)stream;
    if (n == 0) return LIG_OK;
    const double scale = 2.0 / (3.0 * (double)H * (double)W);
    if (dtype == LIG_F32) {
        CotSrc<float> cot{nullptr, nullptr, (const float *)img, (const float *)target,
                          (const float *)grad_loss, (float)scale};
        return raster_bwd<float>(BatchGeo::single(H, W, B, n), TileWalk{}, ids, bins, d_total,
                                 xys, con, col, op, fin, cot,
                                 nullptr, nullptr, nullptr, clamp, ws, ws_bytes, v_xy, v_abs,
                                 v_con, v_rgb, v_op, s);
    }
    if (dtype == LIG_F64) {
        CotSrc<double> cot{nullptr, nullptr, (const double *)img, (const double *)target,
                           (const double *)grad_loss, scale};
        return raster_bwd<double>(BatchGeo::single(H, W, B, n), TileWalk{}, ids, bins, d_total,
                                  xys, con, col, op, fin, cot,
                                  nullptr, nullptr, nullptr, clamp, ws, ws_bytes, v_xy, v_abs,
                                  v_con, v_rgb, v_op, s);
    }
    return LIG_ERR_INVALID;
}

// Number of bounded device-side waits (mbarrier polls of the bulk-staged
// backward) that gave up on the current device since the library loaded;
// 0 unless a kernel malfunctioned.
extern "C" int lig_wait_timeouts(void) {
    unsigned int v = 0;
    if (cudaMemcpyFromSymbol(&v, g_wait_timeouts, sizeof(v)) != cudaSuccess) return -1;
    return (int)v;
}

// ------------------------------------------------------ alpha cut check
namespace lig {
// out[0] = the warp search's cut; out[1] = first failing, out[2] = last
// passing bit pattern of the scan below (initial values for its atomics).
__global__ void alpha_cut_init_kernel(uint32_t *out) {
    const uint32_t cut = alpha_cut_search();
    if (threadIdx.x == 0) {
        out[0] = cut;
        out[1] = 0xffffffffu;
        out[2] = 0u;
    }
}

// The rasterizers' alpha decision at every non-negative float up to +inf
// (bit patterns 0 .. 0x7f800000): the decision is a step with its edge at the
// cut exactly when out[2] + 1 == out[1] == out[0].
__global__ void alpha_cut_scan_kernel(uint32_t *out) {
    constexpr uint32_t kLast = 0x7f800000u;
    uint32_t first_fail = 0xffffffffu, last_pass = 0u;
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u <= kLast; u += stride) {
        if (alpha_passes(__uint_as_float(u))) last_pass = max(last_pass, u);
        else first_fail = min(first_fail, u);
    }
    first_fail = __reduce_min_sync(0xffffffffu, first_fail);
    last_pass = __reduce_max_sync(0xffffffffu, last_pass);
    if ((threadIdx.x & 31) == 0) {
        atomicMin(out + 1, first_fail);
        atomicMax(out + 2, last_pass);
    }
}
}  // namespace lig

// Writes the alpha cut and the full scan's step edges into out[0..2] (device
// memory, three uint32) on `stream`.
extern "C" int lig_alpha_cut(uint32_t *out, void *stream) {
    if (!out) return LIG_ERR_INVALID;
    cudaStream_t s = (cudaStream_t)stream;
    alpha_cut_init_kernel<<<1, 32, 0, s>>>(out);
    alpha_cut_scan_kernel<<<148 * 8, 256, 0, s>>>(out);
    note_launches(2);
    LIG_LAUNCH_CHECK();
    return LIG_OK;
}

// ----------------------------------------------------- allocation-free entry
// Some callers cannot allocate device memory at the time they render: a
// plugin inside a framework that has already reserved (nearly) all of the
// GPU's memory for its own pool, or a real-time loop whose host forbids
// driver allocations after start-up.  For them, the sum forward below takes
// its scratch (the packed per-Gaussian records) from a fixed array compiled
// into this library instead of a caller workspace.  Every GPU that loads the
// library keeps this array (LIG_STATIC_MAX_POINTS records, 6 MiB) until the
// process exits.
namespace lig {
__device__ __align__(256) unsigned char g_noalloc_scratch[(size_t)LIG_STATIC_MAX_POINTS *
                                                          sizeof(Rec<float>)];

// Device address of the scratch array, looked up once per device (host code
// cannot use the symbol itself: on the host it names a stand-in, not device
// memory).  The first call on a device does the lookup.  A device reset by
// the host application (cudaDeviceReset) ends the context the address
// belongs to: each call first checks, with a host-side pointer query, that
// the cached address is still this device's memory, and looks it up again
// when it is not.
static void *noalloc_scratch_ptr(int &rc) {
    static std::mutex mu;
    static void *ptrs[128] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 128) {
        rc = LIG_ERR_LAUNCH;
        return nullptr;
    }
    std::lock_guard<std::mutex> lock(mu);
    if (ptrs[dev]) {
        cudaPointerAttributes a{};
        if (cudaPointerGetAttributes(&a, ptrs[dev]) != cudaSuccess ||
            a.type != cudaMemoryTypeDevice || a.device != dev) {
            (void)cudaGetLastError();  // the failed query must not reach the launch check
            ptrs[dev] = nullptr;
        }
    }
    if (!ptrs[dev]) {
        void *p = nullptr;
        if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || !p) {
            rc = LIG_ERR_LAUNCH;
            return nullptr;
        }
        ptrs[dev] = p;
    }
    rc = LIG_OK;
    return ptrs[dev];
}
}  // namespace lig

extern "C" int lig_raster_fwd_noalloc(int H, int W, int B, int n, const int32_t *ids,
                                      const int32_t *bins, const int32_t *d_total,
                                      const float *xys, const float *con, const float *col,
                                      const float *op, float *img, float *wsum, int32_t *fin,
                                      void *stream) {
    if (n > LIG_STATIC_MAX_POINTS) return LIG_ERR_TOO_LARGE;
    if (!raster_args_ok(H, W, B, n) || !bins || !d_total || !img || !wsum || !fin ||
        (n > 0 && (!xys || !con || !col)))
        return LIG_ERR_INVALID;
    int rc = LIG_OK;
    void *scratch = noalloc_scratch_ptr(rc);
    if (rc != LIG_OK) return rc;
    return raster_fwd<float>(BatchGeo::single(H, W, B, n), TileWalk{}, ids, bins, d_total, xys,
                             con, col, op, scratch, sizeof(g_noalloc_scratch), img, wsum, nullptr,
                             nullptr, nullptr, fin, (cudaStream_t)stream);
}

// ------------------------------------------------------------ batched entries
// A batch of images in one launch per stage: image i has heights[i] x
// widths[i] pixels and counts[i] Gaussians; Gaussians, tile lists and the
// HWC buffers are the images' arrays concatenated in batch order.  The
// (image, tile) work list is flattened (image-major, row-major tiles within
// an image); persistent != 0 runs one CTA per resident slot pulling work
// items from `work` (one int of device memory, overwritten).
namespace lig {
inline bool batch_geo(int n_img, const int32_t *h, const int32_t *w, const int32_t *c, int B,
                      BatchGeo &geo) {
    if (!h || !w || !c || B < 2 || B > 32) return false;
    return BatchGeo::make(n_img, h, w, c, B, geo);
}
}  // namespace lig

extern "C" int lig_raster_fwd_batch(int dtype, int n_img, const int32_t *heights,
                                    const int32_t *widths, const int32_t *counts, int B,
                                    const int32_t *ids, const int32_t *bins,
                                    const int32_t *d_total, const int32_t *cum, const void *xys,
                                    const void *con, const void *col, const void *op,
                                    int persistent, int32_t *work, void *ws, size_t ws_bytes,
                                    void *img, void *wsum, void *dx, void *dy, void *dxy,
                                    int32_t *fin, void *stream) {
    BatchGeo geo;
    if (!batch_geo(n_img, heights, widths, counts, B, geo)) return LIG_ERR_INVALID;
    const int n = geo.total_points();
    if (!bins || !d_total || !img || !wsum || !fin || !ws || (persistent && !work) ||
        (n > 0 && (!xys || !con || !col || !cum)) || ((dx || dy || dxy) && !(dx && dy && dxy)))
        return LIG_ERR_INVALID;
    TileWalk walk{n > 0 ? cum : nullptr, persistent ? work : nullptr};
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype == LIG_F32)
        return raster_fwd<float>(geo, walk, ids, bins, d_total, xys, con, col, op, ws, ws_bytes,
                                 img, wsum, dx, dy, dxy, fin, s);
    if (dtype == LIG_F64)
        return raster_fwd<double>(geo, walk, ids, bins, d_total, xys, con, col, op, ws, ws_bytes,
                                  img, wsum, dx, dy, dxy, fin, s);
    return LIG_ERR_INVALID;
}

extern "C" int lig_views_project(int n_img, const int32_t *heights, const int32_t *widths,
                                 const int32_t *counts, int B, const float *const *in3,
                                 const float *const *means, const float *const *opac,
                                 const float *const *rgb, const int32_t *chol,
                                 const double *origins, const double *scales, void *ws,
                                 size_t ws_bytes, float *xys, float *extents,
                                 int32_t *num_tiles_hit, void *stream) {
    BatchGeo geo;
    if (!in3 || !means || !opac || !rgb || !chol || !origins || !scales ||
        !batch_geo(n_img, heights, widths, counts, B, geo))
        return LIG_ERR_INVALID;
    const int n = geo.total_points();
    if (n > 0 && (!ws || !xys || !extents || !num_tiles_hit)) return LIG_ERR_INVALID;
    if (ws_bytes < sizeof(Rec<float>) * (size_t)n) return LIG_ERR_WORKSPACE;
    if ((reinterpret_cast<uintptr_t>(ws) & 15) != 0) return LIG_ERR_INVALID;  // 16-byte records
    ViewSets sets;
    sets.block_off[0] = 0;
    for (int i = 0; i < n_img; ++i) {
        const double ox = origins[2 * i], oy = origins[2 * i + 1];
        const double sx = scales[2 * i], sy = scales[2 * i + 1];
        if (!(sx > 0.0) || !(sy > 0.0) || !std::isfinite(sx) || !std::isfinite(sy) ||
            !std::isfinite(ox) || !std::isfinite(oy) ||
            (counts[i] > 0 && (!in3[i] || !means[i] || !rgb[i])))
            return LIG_ERR_INVALID;
        sets.block_off[i + 1] = sets.block_off[i] + (counts[i] + 255) / 256;
        sets.v[i] = ViewSet{in3[i],    means[i],  opac[i],   rgb[i], (float)ox,
                            (float)oy, (float)sx, (float)sy, chol[i]};
    }
    if (n == 0) return LIG_OK;
    project_views_kernel<<<sets.block_off[n_img], 256, 0, (cudaStream_t)stream>>>(
        geo, sets, xys, extents, num_tiles_hit, (Rec<float> *)ws);
    note_launches(1);
    LIG_LAUNCH_CHECK();
    return LIG_OK;
}

extern "C" int lig_views_raster(int n_img, const int32_t *heights, const int32_t *widths,
                                const int32_t *counts, int B, const int32_t *ids,
                                const int32_t *bins, const int32_t *cum, int with_opacities,
                                const void *ws, size_t ws_bytes, float *const *imgs,
                                void *stream) {
    BatchGeo geo;
    if (!bins || !cum || !imgs || !batch_geo(n_img, heights, widths, counts, B, geo))
        return LIG_ERR_INVALID;
    const int n = geo.total_points();
    if (n > 0 && (!ids || !ws)) return LIG_ERR_INVALID;
    if (ws_bytes < sizeof(Rec<float>) * (size_t)n) return LIG_ERR_WORKSPACE;
    if ((reinterpret_cast<uintptr_t>(ws) & 15) != 0) return LIG_ERR_INVALID;
    ViewImages out;
    for (int i = 0; i < n_img; ++i) {
        if (!imgs[i]) return LIG_ERR_INVALID;
        out.img[i] = imgs[i];
    }
    // pixels a lane and CTAs per SM as in raster_fwd
    const bool ppl4 = B > 8 && geo.total_tiles() >= LIG_RASTER_PPL4_MIN_TILES;
    const int nt = 32 * Regions::make(ppl4 ? 3 : 1, B).count;
    const size_t sm = (size_t)nt * sizeof(Rec<float>);
    auto pick = [&](auto op_t) {
        constexpr bool O = decltype(op_t)::value;
        return ppl4 ? (nt <= 64 ? raster_views_kernel<4, 64, 16, O> : raster_views_kernel<4, 512, 2, O>)
                    : (nt <= 128 ? raster_views_kernel<2, 128, 9, O>
                                 : raster_views_kernel<2, 512, 2, O>);
    };
    auto fn = with_opacities ? pick(std::true_type{}) : pick(std::false_type{});
    if (!set_dyn_smem((const void *)fn, sm)) return launch_refused();
    fn<<<geo.total_tiles(), nt, sm, (cudaStream_t)stream>>>(
        geo, cum, ids, (const int2 *)bins, (const Rec<float> *)ws, out);
    note_launches(1);
    LIG_LAUNCH_CHECK();
    return LIG_OK;
}

extern "C" int lig_raster_bwd_l2_batch(int dtype, int n_img, const int32_t *heights,
                                       const int32_t *widths, const int32_t *counts, int B,
                                       const int32_t *ids, const int32_t *bins,
                                       const int32_t *d_total, const int32_t *cum,
                                       const void *xys, const void *con, const void *col,
                                       const void *op, const int32_t *fin, const void *img,
                                       const void *target, const void *grad_loss, double clamp,
                                       int persistent, int32_t *work, void *ws, size_t ws_bytes,
                                       void *v_xy, void *v_abs, void *v_con, void *v_rgb,
                                       void *v_op, void *stream) {
    BatchGeo geo;
    if (!batch_geo(n_img, heights, widths, counts, B, geo)) return LIG_ERR_INVALID;
    const int n = geo.total_points();
    if (!bins || !d_total || !fin || !img || !target || !grad_loss || !ws ||
        (persistent && !work) ||
        (n > 0 && (!xys || !con || !col || !cum || !v_xy || !v_abs || !v_con || !v_rgb)))
        return LIG_ERR_INVALID;
    if (n == 0) return LIG_OK;
    TileWalk walk{cum, persistent ? work : nullptr};
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype == LIG_F32) {
        // per-image scale 2 / (3 H_i W_i) is formed in the kernel
        CotSrc<float> cot{nullptr, nullptr, (const float *)img, (const float *)target,
                          (const float *)grad_loss, 0.f};
        return raster_bwd<float>(geo, walk, ids, bins, d_total, xys, con, col, op, fin, cot,
                                 nullptr, nullptr, nullptr, clamp, ws, ws_bytes, v_xy, v_abs,
                                 v_con, v_rgb, v_op, s);
    }
    if (dtype == LIG_F64) {
        CotSrc<double> cot{nullptr, nullptr, (const double *)img, (const double *)target,
                           (const double *)grad_loss, 0.0};
        return raster_bwd<double>(geo, walk, ids, bins, d_total, xys, con, col, op, fin, cot,
                                  nullptr, nullptr, nullptr, clamp, ws, ws_bytes, v_xy, v_abs,
                                  v_con, v_rgb, v_op, s);
    }
    return LIG_ERR_INVALID;
}

// ------------------------------------------------------- fused-L2 forward
// The fit loop's forward: tile lists rendered as lig_raster_fwd, but each
// pixel stores diff = (0 <= x <= 1) ? clamp(x) - target : 0 (not the image)
// and loss = sum_i mean_i((clamp(x) - target)^2) is reduced from per-tile
// fp64 partials; lig_raster_bwd_diff then forms the loss gradient from diff.
extern "C" size_t lig_l2_tile_partials_bytes(int num_tiles) {
    return sizeof(double) * (loss_ticket_offset(num_tiles) + 1);
}

namespace lig {
// target: T values, or bytes when u8
template <typename T>
int fwd_l2(const BatchGeo &geo, TileWalk walk, const int32_t *ids, const int32_t *bins,
           const int32_t *d_total, const void *xys, const void *con, const void *col,
           const void *op, const void *target, void *ws, size_t ws_bytes, double *partials,
           void *diff, int32_t *fin, void *loss, void *per_image, cudaStream_t s,
           bool u8 = false) {
    const L2Fwd<T> l2 = u8 ? L2Fwd<T>{nullptr, partials, (const uint8_t *)target}
                           : L2Fwd<T>{(const T *)target, partials};
    return raster_fwd<T>(geo, walk, ids, bins, d_total, xys, con, col, op, ws, ws_bytes, diff,
                         nullptr, nullptr, nullptr, nullptr, fin, s, l2,
                         L2Out<T>{(T *)loss, (T *)per_image});
}

template <typename T>
int bwd_diff(const BatchGeo &geo, TileWalk walk, const int32_t *ids, const int32_t *bins,
             const int32_t *d_total, const void *xys, const void *con, const void *col,
             const void *op, const int32_t *fin, const void *diff, const void *grad_loss,
             double clamp, void *ws, size_t ws_bytes, void *v_xy, void *v_abs, void *v_con,
             void *v_rgb, void *v_op, cudaStream_t s) {
    // per-image scale 2 / (3 H_i W_i) is formed in the kernel
    CotSrc<T> cot{nullptr, nullptr, nullptr, nullptr, (const T *)grad_loss, (T)0,
                  (const T *)diff};
    return raster_bwd<T>(geo, walk, ids, bins, d_total, xys, con, col, op, fin, cot, nullptr,
                         nullptr, nullptr, clamp, ws, ws_bytes, v_xy, v_abs, v_con, v_rgb, v_op,
                         s);
}
}  // namespace lig

extern "C" int lig_raster_fwd_l2(int dtype, int H, int W, int B, int n, const int32_t *ids,
                                 const int32_t *bins, const int32_t *d_total, const void *xys,
                                 const void *con, const void *col, const void *op,
                                 const void *target, void *ws, size_t ws_bytes,
                                 double *tile_partials, void *diff, int32_t *fin, void *loss,
                                 void *stream) {
    if (!raster_args_ok(H, W, B, n) || !bins || !d_total || !target || !ws || !tile_partials ||
        !diff || !loss || (n > 0 && (!xys || !con || !col)))
        return LIG_ERR_INVALID;
    const BatchGeo geo = BatchGeo::single(H, W, B, n);
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype == LIG_F32)
        return fwd_l2<float>(geo, TileWalk{}, ids, bins, d_total, xys, con, col, op, target, ws,
                             ws_bytes, tile_partials, diff, fin, loss, nullptr, s);
    if (dtype == LIG_F64)
        return fwd_l2<double>(geo, TileWalk{}, ids, bins, d_total, xys, con, col, op, target, ws,
                              ws_bytes, tile_partials, diff, fin, loss, nullptr, s);
    return LIG_ERR_INVALID;
}

extern "C" int lig_raster_fwd_l2_u8(int dtype, int H, int W, int B, int n, const int32_t *ids,
                                    const int32_t *bins, const int32_t *d_total, const void *xys,
                                    const void *con, const void *col, const void *op,
                                    const uint8_t *target, void *ws, size_t ws_bytes,
                                    double *tile_partials, void *diff, int32_t *fin, void *loss,
                                    void *stream) {
    if (!raster_args_ok(H, W, B, n) || !bins || !d_total || !target || !ws || !tile_partials ||
        !diff || !loss || (n > 0 && (!xys || !con || !col)))
        return LIG_ERR_INVALID;
    const BatchGeo geo = BatchGeo::single(H, W, B, n);
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype == LIG_F32)
        return fwd_l2<float>(geo, TileWalk{}, ids, bins, d_total, xys, con, col, op, target, ws,
                             ws_bytes, tile_partials, diff, fin, loss, nullptr, s, true);
    if (dtype == LIG_F64)
        return fwd_l2<double>(geo, TileWalk{}, ids, bins, d_total, xys, con, col, op, target, ws,
                              ws_bytes, tile_partials, diff, fin, loss, nullptr, s, true);
    return LIG_ERR_INVALID;
}

extern "C" int lig_raster_bwd_diff(int dtype, int H, int W, int B, int n, const int32_t *ids,
                                   const int32_t *bins, const int32_t *d_total, const void *xys,
                                   const void *con, const void *col, const void *op,
                                   const int32_t *fin, const void *diff, const void *grad_loss,
                                   double clamp, void *ws, size_t ws_bytes, void *v_xy,
                                   void *v_abs, void *v_con, void *v_rgb, void *v_op,
                                   void *stream) {
    if (!raster_args_ok(H, W, B, n) || !bins || !d_total || (!fin && op) || !diff ||
        !grad_loss || !ws || (n > 0 && (!xys || !con || !col || !v_xy || !v_abs || !v_con || !v_rgb)))
        return LIG_ERR_INVALID;
    if (n == 0) return LIG_OK;
    const BatchGeo geo = BatchGeo::single(H, W, B, n);
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype == LIG_F32)
        return bwd_diff<float>(geo, TileWalk{}, ids, bins, d_total, xys, con, col, op, fin, diff,
                               grad_loss, clamp, ws, ws_bytes, v_xy, v_abs, v_con, v_rgb, v_op, s);
    if (dtype == LIG_F64)
        return bwd_diff<double>(geo, TileWalk{}, ids, bins, d_total, xys, con, col, op, fin,
                                diff, grad_loss, clamp, ws, ws_bytes, v_xy, v_abs, v_con, v_rgb,
                                v_op, s);
    return LIG_ERR_INVALID;
}

extern "C" int lig_raster_fwd_l2_batch(int dtype, int n_img, const int32_t *heights,
                                       const int32_t *widths, const int32_t *counts, int B,
                                       const int32_t *ids, const int32_t *bins,
                                       const int32_t *d_total, const int32_t *cum,
                                       const void *xys, const void *con, const void *col,
                                       const void *op, const void *target, int persistent,
                                       int32_t *work, void *ws, size_t ws_bytes,
                                       double *tile_partials, void *diff, int32_t *fin,
                                       void *loss, void *per_image, void *stream) {
    BatchGeo geo;
    if (!batch_geo(n_img, heights, widths, counts, B, geo)) return LIG_ERR_INVALID;
    const int n = geo.total_points();
    if (!bins || !d_total || !target || !ws || !tile_partials || !diff || !loss ||
        (persistent && !work) || (n > 0 && (!xys || !con || !col || !cum)))
        return LIG_ERR_INVALID;
    TileWalk walk{n > 0 ? cum : nullptr, persistent ? work : nullptr};
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype == LIG_F32)
        return fwd_l2<float>(geo, walk, ids, bins, d_total, xys, con, col, op, target, ws,
                             ws_bytes, tile_partials, diff, fin, loss, per_image, s);
    if (dtype == LIG_F64)
        return fwd_l2<double>(geo, walk, ids, bins, d_total, xys, con, col, op, target, ws,
                              ws_bytes, tile_partials, diff, fin, loss, per_image, s);
    return LIG_ERR_INVALID;
}

extern "C" int lig_raster_fwd_l2_u8_batch(int dtype, int n_img, const int32_t *heights,
                                          const int32_t *widths, const int32_t *counts, int B,
                                          const int32_t *ids, const int32_t *bins,
                                          const int32_t *d_total, const int32_t *cum,
                                          const void *xys, const void *con, const void *col,
                                          const void *op, const uint8_t *target, int persistent,
                                          int32_t *work, void *ws, size_t ws_bytes,
                                          double *tile_partials, void *diff, int32_t *fin,
                                          void *loss, void *per_image, void *stream) {
    BatchGeo geo;
    if (!batch_geo(n_img, heights, widths, counts, B, geo)) return LIG_ERR_INVALID;
    const int n = geo.total_points();
    if (!bins || !d_total || !target || !ws || !tile_partials || !diff || !loss ||
        (persistent && !work) || (n > 0 && (!xys || !con || !col || !cum)))
        return LIG_ERR_INVALID;
    TileWalk walk{n > 0 ? cum : nullptr, persistent ? work : nullptr};
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype == LIG_F32)
        return fwd_l2<float>(geo, walk, ids, bins, d_total, xys, con, col, op, target, ws,
                             ws_bytes, tile_partials, diff, fin, loss, per_image, s, true);
    if (dtype == LIG_F64)
        return fwd_l2<double>(geo, walk, ids, bins, d_total, xys, con, col, op, target, ws,
                              ws_bytes, tile_partials, diff, fin, loss, per_image, s, true);
    return LIG_ERR_INVALID;
}

extern "C" int lig_raster_bwd_diff_batch(int dtype, int n_img, const int32_t *heights,
                                         const int32_t *widths, const int32_t *counts, int B,
                                         const int32_t *ids, const int32_t *bins,
                                         const int32_t *d_total, const int32_t *cum,
                                         const void *xys, const void *con, const void *col,
                                         const void *op, const int32_t *fin, const void *diff,
                                         const void *grad_loss, double clamp, int persistent,
                                         int32_t *work, void *ws, size_t ws_bytes, void *v_xy,
                                         void *v_abs, void *v_con, void *v_rgb, void *v_op,
                                         void *stream) {
    BatchGeo geo;
    if (!batch_geo(n_img, heights, widths, counts, B, geo)) return LIG_ERR_INVALID;
    const int n = geo.total_points();
    if (!bins || !d_total || (!fin && op) || !diff || !grad_loss || !ws || (persistent && !work) ||
        (n > 0 && (!xys || !con || !col || !cum || !v_xy || !v_abs || !v_con || !v_rgb)))
        return LIG_ERR_INVALID;
    if (n == 0) return LIG_OK;
    TileWalk walk{cum, persistent ? work : nullptr};
    cudaStream_t s = (cudaStream_t)stream;
    if (dtype == LIG_F32)
        return bwd_diff<float>(geo, walk, ids, bins, d_total, xys, con, col, op, fin, diff,
                               grad_loss, clamp, ws, ws_bytes, v_xy, v_abs, v_con, v_rgb, v_op, s);
    if (dtype == LIG_F64)
        return bwd_diff<double>(geo, walk, ids, bins, d_total, xys, con, col, op, fin, diff,
                                grad_loss, clamp, ws, ws_bytes, v_xy, v_abs, v_con, v_rgb, v_op,
                                s);
    return LIG_ERR_INVALID;
}

// ------------------------------------------------------------------ fit step
// The fit engine's iteration, with what its seven separate calls repeat taken
// out: the projection writes the forward's records, which serve the backward,
// and clears what the later launches start from; the loss launch forms Adam's scalars and mirrors the skip count, and one
// kernel takes the backward's packed sums through the projection backward and
// Adam.  64 B of parameters and gradients, 128 B of moments and the 32 B sums
// move once per Gaussian; before, v_xy, v_conic and the gradients were written
// and read again between five launches.  Iteration: 512^2 / 50k 121 -> 96 us (12
// launches instead of 21), 16 images 875 -> 847, 2048^2 / 1M 1497 -> 1458, 8192^2 /
// 2M 3736 -> 3662.
namespace lig {
__global__ void __launch_bounds__(256)
fit_update_kernel(const BatchGeo geo, int n, const float4 *__restrict__ packed,
                  float *__restrict__ p, float *__restrict__ g, float *__restrict__ m,
                  float *__restrict__ v, float c1, float b2, float c2, float eps,
                  const AdamScalars *__restrict__ sc) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 q0 = packed[2 * (size_t)i], q1 = packed[2 * (size_t)i + 1];
    const float v_xy[2] = {q0.x, q0.y}, v_con[3] = {q0.z, q0.w, q1.x};
    const size_t at[8] = {2 * (size_t)i, 2 * (size_t)i + 1,
                          2 * (size_t)n + 3 * (size_t)i, 2 * (size_t)n + 3 * (size_t)i + 1,
                          2 * (size_t)n + 3 * (size_t)i + 2,
                          5 * (size_t)n + 3 * (size_t)i, 5 * (size_t)n + 3 * (size_t)i + 1,
                          5 * (size_t)n + 3 * (size_t)i + 2};
    float gr[8];
    project_vjp<float>(geo, true, p + 2 * (size_t)n, p, nullptr, i, v_xy, v_con, gr[2], gr[3],
                       gr[4], gr[0], gr[1]);
    gr[5] = q1.y;
    gr[6] = q1.z;
    gr[7] = q1.w;
#pragma unroll
    for (int k = 0; k < 8; ++k) g[at[k]] = gr[k];
    const AdamScalars a = sc[geo.image_of_gauss(i)];
    if (a.skip) return;
    float pe[8], me[8], ve[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        pe[k] = p[at[k]];
        me[k] = m[at[k]];
        ve[k] = v[at[k]];
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        adam_update(pe[k], gr[k], me[k], ve[k], c1, b2, c2, eps, a);
        p[at[k]] = pe[k];
        m[at[k]] = me[k];
        v[at[k]] = ve[k];
    }
}
}  // namespace lig

extern "C" int lig_fit_bin_batch(int n_img, const int32_t *heights, const int32_t *widths,
                                 const int32_t *counts, int B, const float *params, void *ws,
                                 size_t ws_bytes, double *tile_partials, float *xys,
                                 float *extents, int32_t *num_tiles_hit, int32_t *cum,
                                 int32_t *d_total, void *cum_ws, size_t cum_ws_bytes, int capacity,
                                 void *bin_ws, size_t bin_ws_bytes, int32_t *ids, int32_t *bins,
                                 int32_t *status, void *stream) {
    BatchGeo geo;
    if (!batch_geo(n_img, heights, widths, counts, B, geo)) return LIG_ERR_INVALID;
    const int n = geo.total_points();
    if (capacity < 0 || !ws || !tile_partials || !d_total || !bins || !status ||
        (capacity > 0 && (!ids || !bin_ws)) ||
        (n > 0 && (!params || !xys || !extents || !num_tiles_hit || !cum || !cum_ws)) ||
        (reinterpret_cast<uintptr_t>(ws) & 15) != 0 ||      // 16-byte records
        (reinterpret_cast<uintptr_t>(cum_ws) & 7) != 0)
        return LIG_ERR_INVALID;
    const size_t goff = bwd_grad_offset<float>(n);
    if (ws_bytes < goff + sizeof(float) * 8 * (size_t)n ||
        (n > 0 && cum_ws_bytes < lig_cumsum_workspace_bytes(n)))
        return LIG_ERR_WORKSPACE;
    cudaStream_t s = (cudaStream_t)stream;
    uint32_t *ticket = loss_ticket(tile_partials, geo.total_tiles());
    if (n == 0) {
        cudaMemsetAsync(ticket, 0, sizeof(*ticket), s);
        cudaMemsetAsync(status, 0, sizeof(*status), s);
    } else {
        fit_project_kernel<<<(n + 255) / 256, 256, 0, s>>>(
            geo, n, params, xys, extents, num_tiles_hit, (Rec<float> *)ws,
            (float4 *)((char *)ws + goff), (uint32_t *)cum_ws,
            (int)(lig_cumsum_workspace_bytes(n) / sizeof(uint32_t)), status, ticket);
        note_launches(1);
        LIG_LAUNCH_CHECK();
    }
    return scan_and_bin(geo, xys, extents, num_tiles_hit, cum, d_total, cum_ws, capacity, bin_ws,
                        bin_ws_bytes, ids, bins, status, s);
}

extern "C" int lig_fit_forward_batch(int n_img, const int32_t *heights, const int32_t *widths,
                                     const int32_t *counts, int B, const int32_t *ids,
                                     const int32_t *bins, const int32_t *d_total,
                                     const int32_t *cum, const void *target, int target_u8,
                                     int persistent, int32_t *work, void *ws, size_t ws_bytes,
                                     double *tile_partials, float *diff, float *loss,
                                     float *per_image, const int32_t *status, int32_t *steps,
                                     int32_t *skipped, int32_t *skipped_host, double lr,
                                     double beta1, double beta2, void *scratch,
                                     size_t scratch_bytes, void *stream) {
    BatchGeo geo;
    if (!batch_geo(n_img, heights, widths, counts, B, geo)) return LIG_ERR_INVALID;
    const int n = geo.total_points();
    if (!bins || !d_total || !target || !ws || !tile_partials || !diff || !loss || !status ||
        !steps || !skipped || !skipped_host || !scratch || (persistent && !work) ||
        (n > 0 && !cum))
        return LIG_ERR_INVALID;
    const size_t goff = bwd_grad_offset<float>(n);
    if (ws_bytes < goff + sizeof(float) * 8 * (size_t)n ||
        scratch_bytes < sizeof(AdamScalars) * (size_t)n_img)
        return LIG_ERR_WORKSPACE;
    const L2Fwd<float> l2 =
        target_u8 ? L2Fwd<float>{nullptr, tile_partials, (const uint8_t *)target}
                  : L2Fwd<float>{(const float *)target, tile_partials};
    TileWalk walk{n > 0 ? cum : nullptr, persistent ? work : nullptr};
    return raster_fwd<float>(geo, walk, ids, bins, d_total, nullptr, nullptr, nullptr, nullptr, ws,
                             goff, diff, nullptr, nullptr, nullptr, nullptr, nullptr,
                             (cudaStream_t)stream, l2, L2Out<float>{loss, per_image}, true,
                             AdamPro{status, steps, skipped, skipped_host, lr, beta1, beta2,
                                     (AdamScalars *)scratch});
}

extern "C" int lig_fit_backward_batch(int n_img, const int32_t *heights, const int32_t *widths,
                                      const int32_t *counts, int B, const int32_t *ids,
                                      const int32_t *bins, const int32_t *d_total,
                                      const int32_t *cum, const float *diff,
                                      const float *grad_loss, int persistent, int32_t *work,
                                      void *ws, size_t ws_bytes, float *params, float *grads,
                                      float *exp_avg, float *exp_avg_sq, double beta1,
                                      double beta2, double eps, const void *scratch,
                                      void *stream) {
    BatchGeo geo;
    if (!batch_geo(n_img, heights, widths, counts, B, geo)) return LIG_ERR_INVALID;
    const int n = geo.total_points();
    if (!bins || !d_total || !diff || !grad_loss || !ws || !scratch || (persistent && !work) ||
        (n > 0 && (!cum || !params || !grads || !exp_avg || !exp_avg_sq)))
        return LIG_ERR_INVALID;
    if (n == 0) return LIG_OK;
    cudaStream_t s = (cudaStream_t)stream;
    TileWalk walk{cum, persistent ? work : nullptr};
    CotSrc<float> cot{nullptr, nullptr, nullptr, nullptr, grad_loss, 0.f, diff};
    int rc = raster_bwd<float>(geo, walk, ids, bins, d_total, nullptr, nullptr, nullptr, nullptr,
                               nullptr, cot, nullptr, nullptr, nullptr, 0.0, ws, ws_bytes, nullptr,
                               nullptr, nullptr, nullptr, nullptr, s, /*prepacked=*/true);
    if (rc) return rc;
    const float *packed = (const float *)((char *)ws + bwd_grad_offset<float>(n));
    fit_update_kernel<<<(n + 255) / 256, 256, 0, s>>>(
        geo, n, (const float4 *)packed, params, grads, exp_avg, exp_avg_sq, (float)(1.0 - beta1),
        (float)beta2, (float)(1.0 - beta2), (float)eps, (const AdamScalars *)scratch);
    note_launches(1);
    LIG_LAUNCH_CHECK();
    return LIG_OK;
}
