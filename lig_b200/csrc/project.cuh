// Per-Gaussian projection math shared by the projection kernels and the fused
// fit step.
#pragma once
#include "common.cuh"

namespace lig {

// Optional view transform of a render (region decode, scale_to): output
// pixel coordinates are ((x - ox) sx, (y - oy) sy) in the Gaussians' frame,
// so every Gaussian maps to means' = (means - origin) * (sx, sy) and
// L' = diag(sx, sy) L (Cholesky; the scale_to rule of
// minimal_trainer_upscale.py:139-157) or cov' = S cov S.  Off: inputs are used
// as they are.
template <typename T> struct View {
    T ox, oy, sx, sy;
    bool on;
};

// cov2d (a,b,c) from the input triple: pass-through, or the Cholesky product
// [l11^2, l11 l21, l21^2 + l22^2] written as in csrc/forward.cu:79-83.
// VIEW is a template parameter so that the plain projection compiles to
// exactly the reference's arithmetic (a runtime branch changes how the
// compiler contracts the products below, and with it the rounding).
template <typename T, bool VIEW = false>
__device__ __forceinline__ void input_cov(bool chol, const T *in3, int i, T &cx, T &cy, T &cz,
                                          const View<T> &v = View<T>{0, 0, 1, 1, false}) {
    T p = in3[3 * i], q = in3[3 * i + 1], r = in3[3 * i + 2];
    if constexpr (VIEW) {
        if (chol) { p *= v.sx; q *= v.sy; r *= v.sy; }
        else { p *= v.sx * v.sx; q *= v.sx * v.sy; r *= v.sy * v.sy; }
    }
    if (chol) {
        cx = p * p;
        cy = p * q;
        cz = q * q + r * r;
    } else {
        cx = p; cy = q; cz = r;
    }
}

// conic VJP (csrc/helpers.cuh:101-110): v_Sigma = -X G X for symmetric X
// (conic) and G (v_conic with halved off-diagonal), written out as the
// column-major 2x2 products in the same evaluation order.
template <typename T>
__device__ __forceinline__ void conic_vjp(T a, T b, T c, T va, T vb, T vc, T &oa, T &ob, T &oc) {
    T g01 = vb / (T)2;
    // N = -X
    T n00 = -a, n01 = -b, n10 = -b, n11 = -c;
    // P = N * G  (P[col][row] = N[0][row]*G[col][0] + N[1][row]*G[col][1])
    T p00 = n00 * va + n10 * g01;
    T p01 = n01 * va + n11 * g01;
    T p10 = n00 * g01 + n10 * vc;
    T p11 = n01 * g01 + n11 * vc;
    // Q = P * X
    T q00 = p00 * a + p10 * b;
    T q01 = p01 * a + p11 * b;
    T q10 = p00 * b + p10 * c;
    T q11 = p01 * b + p11 * c;
    oa = q00;
    ob = q10 + q01;
    oc = q11;
}

// Cholesky chain rule with non-finite -> 0 (csrc/backward.cu:228-246).
template <typename T>
__device__ __forceinline__ void chol_chain(T l11, T l21, T l22, T va, T vb, T vc, T &g11, T &g21,
                                           T &g22) {
    using M = Math<T>;
    T a = (T)2 * l11 * va + l21 * vb;
    T b = l11 * vb + (T)2 * l21 * vc;
    T c = (T)2 * l22 * vc;
    bool fin = M::finite_(a) & M::finite_(b) & M::finite_(c);
    g11 = fin ? a : (T)0;
    g21 = fin ? b : (T)0;
    g22 = fin ? c : (T)0;
}

// Projection backward of Gaussian i from its (v_xy, v_conic), recomputing conic,
// extent and bbox: the validity test (extents > 0 in csrc/backward.cu:195, :217)
// is re-derived exactly because the forward math is re-run with the same code.
template <typename T>
__device__ __forceinline__ void project_vjp(const BatchGeo &geo, bool chol, const T *in3,
                                            const T *means, const T *opac, int i, const T *v_xy,
                                            const T *v_conic, T &o0, T &o1, T &o2, T &m0, T &m1) {
    const int im = geo.image_of_gauss(i);
    const unsigned tbx = geo.tbx[im], tby = geo.tby(im), block = geo.B;
    T cx, cy, cz;
    input_cov(chol, in3, i, cx, cy, cz);
    T o = opac ? opac[i] : (T)1;
    T ca = 0, cb = 0, cc = 0, ex = 0, ey = 0;
    bool valid = cov2d_bounds(cx, cy, cz, o, ca, cb, cc, ex, ey);
    if (valid) {
        int x0, y0, x1, y1;
        tile_bbox(means[2 * i], means[2 * i + 1], ex, ey, tbx, tby, block, x0, y0, x1, y1);
        int32_t area = (int32_t)((unsigned)(x1 - x0) * (unsigned)(y1 - y0));
        valid = area > 0 && ex > (T)0 && ey > (T)0;
    }
    o0 = o1 = o2 = m0 = m1 = 0;
    if (valid) {
        m0 = v_xy[0];
        m1 = v_xy[1];
        T va, vb, vc;
        conic_vjp(ca, cb, cc, v_conic[0], v_conic[1], v_conic[2], va, vb, vc);
        if (chol)
            chol_chain(in3[3 * i], in3[3 * i + 1], in3[3 * i + 2], va, vb, vc, o0, o1, o2);
        else {
            o0 = va; o1 = vb; o2 = vc;
        }
    }
}

}  // namespace lig
