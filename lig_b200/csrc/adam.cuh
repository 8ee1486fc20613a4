// Adam's update rule and its per-step scalars, shared by the optimiser kernels
// and the fused fit step.
#pragma once
#include "common.cuh"

namespace lig {

struct AdamScalars {
    float step_size;     // lr / (1 - b1^t)
    float bc2_sqrt;      // sqrt(1 - b2^t)
    int skip;            // 1: leave everything unchanged
    int pad;
};

// One element, in the form torch.optim.Adam evaluates it: m = lerp(m, g,
// 1 - b1), v = v b2 + (1 - b2) g g, p -= step_size * m / (sqrt(v) / bc2 +
// eps), with correctly rounded square root and divisions.
// c1 = 1 - b1 and c2 = 1 - b2 are formed in double on the host and rounded
// once, as torch does with its Python-float coefficients.
__device__ __forceinline__ void adam_update(float &p, float g, float &m, float &v, float c1,
                                            float b2, float c2, float eps,
                                            const AdamScalars &a) {
    m = __fadd_rn(m, __fmul_rn(c1, __fsub_rn(g, m)));
    v = __fadd_rn(__fmul_rn(v, b2), __fmul_rn(__fmul_rn(c2, g), g));
    const float den = __fadd_rn(__fdiv_rn(__fsqrt_rn(v), a.bc2_sqrt), eps);
    p = __fsub_rn(p, __fmul_rn(a.step_size, __fdiv_rn(m, den)));
}

// A batch of fits in one flat buffer laid out [means 2N | cholesky 3N |
// rgb 3N] (N = total Gaussians, image i owning Gaussians [g_off[i],
// g_off[i+1])).  Every image keeps its own step count, so a fit that joins
// or leaves a running batch follows exactly the updates it would get alone.
struct AdamBatch {
    int n_img, n_pts;
    int g_off[kMaxBatch + 1];
};

// The step's scalars of image i (a thread each, i < n_img): counts the step, or
// — when this step's binning overflowed — marks it skipped (image 0 counts it).
__device__ __forceinline__ void adam_prologue(int i, int n_img, const int32_t *status,
                                              int32_t *steps, int32_t *skipped, double lr,
                                              double b1, double b2, AdamScalars *out) {
    const bool skip = status && (*status & LIG_STATUS_OVERFLOW);
    if (i == 0 && skip && skipped) *skipped += 1;
    if (i >= n_img) return;
    AdamScalars a{0.f, 1.f, skip ? 1 : 0, 0};
    if (!skip) {
        const int t = steps[i] + 1;
        steps[i] = t;
        a.step_size = (float)(lr / (1.0 - pow(b1, (double)t)));
        a.bc2_sqrt = (float)sqrt(1.0 - pow(b2, (double)t));
    }
    out[i] = a;
}

}  // namespace lig
