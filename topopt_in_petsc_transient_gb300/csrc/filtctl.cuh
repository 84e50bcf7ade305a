// filtctl.cuh -- the scalars that steer the PDE filter's solve (filter.cu), formed
// alike by one thread of every CTA, and by the host's check of the same loop.
#pragma once
#include <cmath>

#include "../../include/topopt_gb300.h"

namespace topo {

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

// FP64 from the start?  rho = max_a (R / h_a)^2 is the size of K's entries against
// its row sums.  A correction gains a factor of about 1e6 / rho, and b - K u resolves
// about 3e-16 rho of b, so past either line the corrections only come before the CG
// that they leave the solve to.  Measured, corrections against FP64 CG at rtol 1e-10:
// rho = 2e4 (512 elements) 3.0 against 2.7 ms at 48x24x24, 9.6 : 12.2 at 96x48x48 and
// 47 : 85 at 192x96x96; rho = 8e4 3.2 : 2.8, 11.9 : 12.8 and 58 : 88; at 3.5e5 they
// end unsolved after 1500 iterations.
inline bool filt_in_fp64(const double h[3], double R, double tol) {
    const double hm = fmin(h[0], fmin(h[1], h[2])), rho = R / hm * (R / hm);
    return rho > fmin(1e5, 1e15 * fabs(tol));
}

struct FiltRhs {
    double bb, rr, rms;  // b.b, r.r of the FP64 residual, its root mean square
    float gam, alpha, beta, goal;
    int done, idle;  // solved; no further iteration of this correction
    int hard;        // left to FP64 (FiltCg)
};

// first step of a correction from its sums r.z and w.z
__host__ __device__ inline void filt_begin(FiltRhs &q, float rz, float wz, double tol, long long nn) {
    q.idle = q.done || q.hard;
    if (q.idle) return;
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
// After a correction, from the FP64 residual's r.r.  A correction that does not
// halve the residual is at what FP32, or b - K u itself, can resolve; the next one
// would start where this one did.
__host__ __device__ inline void filt_judge(FiltRhs &q, double rr, double tol, int its, int maxit) {
    if (q.done || q.hard) return;
    const double was = q.rr;
    q.rr = rr;
    if (rr <= tol * tol * q.bb) q.done = 1;
    else if (its >= maxit || !(rr <= 0.25 * was)) q.hard = 1;
}

// Jacobi CG in FP64 from u = 0, which has the last word on what FP32 leaves over:
// it ends on its recurrence's residual or with the status of the solve
struct FiltCg {
    double rz, alpha, beta;
    int it, done, status;
};
__host__ __device__ inline void filt_cg_begin(FiltCg &c, double rz) { c = FiltCg{rz, 0.0, 0.0, 0, 0, TOPO_OK}; }
// after the product, from p.q
__host__ __device__ inline void filt_cg_step(FiltCg &c, double pq) {
    c.alpha = c.rz / pq;
    if (!(pq > 0.0)) {
        c.done = 1;
        c.status = isfinite(pq) ? TOPO_ERR_BREAKDOWN : TOPO_ERR_NAN;
    }
}
// after the update, from r.r and r.z
__host__ __device__ inline void filt_cg_judge(FiltCg &c, double rr, double rz, double tol, double bb, int maxit) {
    c.beta = rz / c.rz;
    c.rz = rz;
    c.it++;
    c.done = 1;
    if (!isfinite(rr)) c.status = TOPO_ERR_NAN;
    else if (rr <= tol * tol * bb) c.status = TOPO_OK;
    else if (c.it >= maxit) c.status = TOPO_ERR_NOT_CONVERGED;
    else c.done = 0;
}

}  // namespace topo
