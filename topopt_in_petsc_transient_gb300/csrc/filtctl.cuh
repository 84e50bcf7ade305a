// filtctl.cuh -- the scalars that steer the PDE filter's solve (filter.cu), formed
// alike by one thread of every CTA, and by the host's check of the same loop.
#pragma once
#include <cmath>

#include "../../include/topopt_gb300.h"

namespace topo {

constexpr int FILT_CAP = 64;  // iterations of a correction

// weights of A (FiltOp, filter.cu) for element edges h and length scale R: c[S] of a
// neighbour displaced along the axes in S
inline void filt_stencil(const double h[3], double R, double c[8]) {
    const double m[2] = {4.0 / 6.0, 1.0 / 6.0}, k[2] = {2.0, -1.0};  // own node, a neighbour
    for (int S = 0; S < 8; S++) {
        const int b[3] = {S & 1, (S >> 1) & 1, S >> 2};
        c[S] = m[b[0]] * m[b[1]] * m[b[2]];
        for (int a = 0; a < 3; a++) c[S] += R * R / (h[a] * h[a]) * k[b[a]] * m[b[(a + 1) % 3]] * m[b[(a + 2) % 3]];
    }
}

struct FiltRhs {
    double bb, rr, rms;  // b.b, r.r of the FP64 residual, its root mean square
    float gam, alpha, beta, goal;
    int done, idle;  // solved; no further iteration of this correction
};

// first step of a correction from its sums r.z and w.z
__host__ __device__ inline void filt_begin(FiltRhs &q, float rz, float wz, double tol, long long nn) {
    q.idle = q.done;
    if (q.done) return;
    q.gam = rz;
    q.beta = 0.0f;
    q.alpha = rz / wz;
    if (!(q.alpha > 0.0f) || !isfinite(q.alpha)) q.idle = 1;
    // reduction asked of this correction: half of what is left to the
    // tolerance, at most 1e-6 (what the FP32 recurrence holds)
    const double left = fmax(1e-6, 0.5 * tol * sqrt(q.bb / q.rr));
    q.goal = (float)(left * left * (double)nn);
}
// after an iteration, from its sums r.z, w.z and r.r
__host__ __device__ inline void filt_advance(FiltRhs &q, const float t[3]) {
    if (q.idle) return;
    const float be = t[0] / q.gam;
    q.beta = be;
    q.alpha = t[0] / (t[1] - be * t[0] / q.alpha);
    q.gam = t[0];
    // at the goal, or rounding has used the correction up
    if (!(t[2] > q.goal) || !(q.alpha > 0.0f) || !isfinite(q.alpha)) q.idle = 1;
}
// after a correction, from the FP64 residual's r.r: status of the solve
__host__ __device__ inline int filt_judge(FiltRhs &q, double rr, double tol, int its, int maxit) {
    if (q.done) return TOPO_OK;
    const double was = q.rr;
    q.rr = rr;
    if (!isfinite(rr)) return TOPO_ERR_NAN;
    // a residual that a correction no longer halves, below 1e-12, is the
    // rounding of b - K u: tolerances under it are met as far as FP64 goes
    if (rr <= tol * tol * q.bb || (rr > 0.25 * was && rr <= 1e-24 * q.bb)) q.done = 1;
    // a correction that leaves the residual where it was leaves the next one nothing
    // else to start from: FP32 cannot solve this system, and `its` need not have moved
    else if (its >= maxit || !(rr < was)) return TOPO_ERR_NOT_CONVERGED;
    return TOPO_OK;
}

}  // namespace topo
