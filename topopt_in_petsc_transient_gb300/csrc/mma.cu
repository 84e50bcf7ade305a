// mma.cu -- the Method of Moving Asymptotes (MMA.cc) with design vectors
// resident on the GPU.
//
// Per design iteration one cooperative kernel (k_mma_update): GenSub
// (MMA.cc:510-637) and the epsilon/Newton loops of SolveDIP (:639-676), one
// pass over the elements per Newton step for the dual's gradient, Hessian and
// residual; the m-sized dual algebra (Hessian corrections, the m x m LU of
// Factorize/Solve, line search) runs in FP64 in one thread of every CTA.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "coop.cuh"
#include "kernels.cuh"
#include "mma.h"

namespace topo {

constexpr int MMA_MAXM = 8;

#define MCK(call)                                                            \
    do {                                                                     \
        cudaError_t e_ = (call);                                             \
        if (e_ != cudaSuccess) {                                             \
            set_error(std::string(#call) + ": " + cudaGetErrorString(e_));  \
            return TOPO_ERR_CUDA;                                            \
        }                                                                    \
    } while (0)

struct MMAScalars {
    int m, k;
    double asyminit, asymdec, asyminc;
    double a[MMA_MAXM], c[MMA_MAXM], d[MMA_MAXM];
    double b[MMA_MAXM], y[MMA_MAXM], z, lam[MMA_MAXM], mu[MMA_MAXM];
    double epsi, err;
};

constexpr int MMA_NT = 256;

// per-element data of one update.  Of the subproblem of an element,
//   min p / (U - x) + q / (x - L),  p = p0 + lam . pij, q = q0 + lam . qij,
// the passes use, with w = U - L: rw = 1 / w, the bounds from L (al = alpha -
// L, be = beta - L) and the constraint's terms at the two bounds (ga, gb).
struct MMAVecs {
    double *L, *U, *p0, *q0, *pij, *qij, *w, *rw, *al, *be, *ga, *gb, *xo1, *xo2;
};
struct MMAArgs {
    long long n;
    MMAVecs v;
    double *x;  // design: xval in, the update out
    const double *dfdx, *dgdx, *xmin, *xmax;
    double gx[MMA_MAXM];
    MMAScalars *S;
    int k;        // iteration number, from 1
    double tol;   // final epsilon
    double *part;  // [2 slots][5 values][gridDim]
    GridBar bar;
    int *status;  // mapped host memory
};

struct TopoMMA {
    int n, m;
    MMAVecs v;
    MMAScalars *S;
    double *part;
    unsigned int *counter;  // [0] reductions, [1..3] the grid barrier
    unsigned long long *bits;
    int *status, *status_dev;  // mapped host memory
    unsigned grid;             // CTAs of k_mma_update: resident at once, at most one per MMA_NT elements
    std::vector<void *> ptrs;
    cudaStream_t stream;
    MMAScalars host;
};

// the dual's state, the same in every CTA
template <int M>
struct MMADual {
    double lam[M], mu[M], y[M], b[M], grad[M], z, epsi, err;
    double G[M], H[M * M];  // sums of DualGrad and DualHess at lam
    int go;                 // another Newton step
};

// scalar part of XYZofLAMBDA (MMA.cc:696-703)
template <int M>
__device__ void mma_yz(MMADual<M> &D, const MMAScalars *S) {
    double lamai = 0.0;
    for (int i = 0; i < M; i++) {
        if (D.lam[i] < 0.0) D.lam[i] = 0;
        D.y[i] = fmax(0.0, D.lam[i] - S->c[i]);
        lamai += D.lam[i] * S->a[i];
    }
    D.z = fmax(0.0, 10.0 * (lamai - 1.0));
}

// Newton step of SolveDIP (MMA.cc:658-670) from the sums at lam
template <int M>
__device__ void mma_newton(MMADual<M> &D, const MMAScalars *S) {
    double *g = D.grad, *H = D.H, st[2 * M];
    for (int j = 0; j < M; j++) {
        g[j] = D.G[j] - D.b[j] - S->a[j] * D.z - D.y[j];
        g[j] = -1.0 * g[j] - D.epsi / D.lam[j];
    }
    // DualHess corrections (MMA.cc:829-858)
    double lamai = 0.0;
    for (int j = 0; j < M; j++) {
        if (D.lam[j] < 0.0) D.lam[j] = 0.0;
        lamai += D.lam[j] * S->a[j];
        if (D.lam[j] > S->c[j]) H[j * M + j] += -1.0;
        H[j * M + j] += -D.mu[j] / D.lam[j];
    }
    if (lamai > 0.0)
        for (int j = 0; j < M; j++)
            for (int kk = 0; kk < M; kk++) H[j * M + kk] += -10.0 * S->a[j] * S->a[kk];
    double tr = 0.0;
    for (int j = 0; j < M; j++) tr += H[j * M + j];
    double corr = 1e-4 * tr / M;
    if (-1.0 * corr < 1.0e-7) corr = -1.0e-7;
    for (int j = 0; j < M; j++) H[j * M + j] += corr;
    // Factorize / Solve (MMA.cc:936-969)
    for (int ss = 0; ss < M - 1; ss++)
        for (int ii = ss + 1; ii < M; ii++) {
            H[ii * M + ss] = H[ii * M + ss] / H[ss * M + ss];
            for (int jj = ss + 1; jj < M; jj++) H[ii * M + jj] = H[ii * M + jj] - H[ii * M + ss] * H[ss * M + jj];
        }
    for (int ii = 1; ii < M; ii++) {
        double aa = 0.0;
        for (int jj = 0; jj < ii; jj++) aa = aa - H[ii * M + jj] * g[jj];
        g[ii] = g[ii] + aa;
    }
    g[M - 1] = g[M - 1] / H[(M - 1) * M + (M - 1)];
    for (int ii = M - 2; ii >= 0; ii--) {
        double aa = g[ii];
        for (int jj = ii + 1; jj < M; jj++) aa = aa - H[ii * M + jj] * g[jj];
        g[ii] = aa / H[ii * M + ii];
    }
    for (int j = 0; j < M; j++) st[j] = g[j];
    for (int j = 0; j < M; j++) st[M + j] = -D.mu[j] + D.epsi / D.lam[j] - st[j] * D.mu[j] / D.lam[j];
    // DualLineSearch (MMA.cc:870-888)
    double theta = 1.005;
    for (int j = 0; j < M; j++) {
        if (theta < -1.01 * st[j] / D.lam[j]) theta = -1.01 * st[j] / D.lam[j];
        if (theta < -1.01 * st[j + M] / D.mu[j]) theta = -1.01 * st[j + M] / D.mu[j];
    }
    theta = 1.0 / theta;
    for (int j = 0; j < M; j++) {
        D.lam[j] = D.lam[j] + theta * st[j];
        D.mu[j] = D.mu[j] + theta * st[j + M];
    }
    mma_yz(D, S);  // XYZofLAMBDA for the new lambda
}

// DualResidual (MMA.cc:890-934) from the sums at lam
template <int M>
__device__ double mma_residual(const MMADual<M> &D, const MMAScalars *S) {
    double nrI = 0.0;
    for (int j = 0; j < M; j++) {
        const double r1 = D.G[j] - D.b[j] - S->a[j] * D.z - D.y[j] + D.mu[j];
        const double r2 = D.mu[j] * D.lam[j] - D.epsi;
        nrI = fmax(nrI, fmax(fabs(r1), fabs(r2)));
    }
    return nrI;
}

// Sums of the dual at lam over this thread's elements: acc = [gradient m |
// upper Hessian].  With sp = sqrt(p), sq = sqrt(q), s = sp + sq the minimiser
// is x = L + w sq / s (MMA.cc:706-712), U - x = w sp / s and x - L = w sq / s,
// so an element strictly between its bounds adds
//   pij / (U - x) + qij / (x - L) = (s / w) (pij / sp + qij / sq)      to the gradient (:738-743) and
//   PQ_j df2 PQ_k = -(1 / 2w) e_j e_k sp sq, e = pij / p - qij / q     to the Hessian (:790-818);
// one at a bound adds ga or gb to the gradient.  About 40 FP64 instructions an
// element against about 200 with a quotient for every term in two passes a
// step, at GB300's 2 lanes a clock and SM the whole time of a pass: an update
// of 1,769,472 elements takes 1.85 ms instead of 6.3, one of 27,648 (launches and
// host polls before) 0.21 instead of 0.59.
template <int M>
__device__ __forceinline__ void mma_sums(const MMAArgs &A, const double *lam, double *acc) {
    const long long n = A.n;
    const MMAVecs &v = A.v;
#pragma unroll
    for (int j = 0; j < M + M * (M + 1) / 2; j++) acc[j] = 0.0;
    for (long long i = blockIdx.x * (long long)MMA_NT + threadIdx.x; i < n; i += (long long)gridDim.x * MMA_NT) {
        double p = v.p0[i], q = v.q0[i], pj[M], qj[M];
        const double w = v.w[i], rw = v.rw[i], al = v.al[i], be = v.be[i];
#pragma unroll
        for (int j = 0; j < M; j++) {
            pj[j] = v.pij[(long long)j * n + i];
            qj[j] = v.qij[(long long)j * n + i];
            p += pj[j] * lam[j];
            q += qj[j] * lam[j];
        }
        const double rp = rsqrt(p), rq = rsqrt(q), sp = p * rp, sq = q * rq, s = sp + sq, t = w * sq;
        const bool low = t < al * s, high = t > be * s;
        if (low || high) {  // x < alpha takes alpha, then x > beta takes beta (MMA.cc:713-716)
            const double *at = (high || al > be) ? v.gb : v.ga;
#pragma unroll
            for (int j = 0; j < M; j++) acc[j] += at[(long long)j * n + i];
            continue;
        }
        double e[M];
        const double c = s * rw, h = -0.5 * rw * (sp * sq);
#pragma unroll
        for (int j = 0; j < M; j++) {
            const double a = pj[j] * rp, b = qj[j] * rq;
            acc[j] += c * (a + b);
            e[j] = a * rp - b * rq;
        }
        int o = M;
#pragma unroll
        for (int a = 0; a < M; a++)
#pragma unroll
            for (int b = a; b < M; b++) acc[o++] += e[a] * (h * e[b]);
    }
}

template <int M>
static __global__ void __launch_bounds__(MMA_NT, 4) k_mma_update(const MMAArgs A) {
    constexpr int NV = M + M * (M + 1) / 2;
    __shared__ double sred[NV * MMA_NT], stot[NV];
    __shared__ MMADual<M> D;
    const MMAScalars *S = A.S;
    const long long n = A.n, t0 = blockIdx.x * (long long)MMA_NT + threadIdx.x, ts = (long long)gridDim.x * MMA_NT;
    unsigned arrivals = 0;
    int slot = 0;
    auto reduce = [&](const double *acc, int nv) {  // grid sums of the first nv values into stot
        double *part = A.part + (size_t)slot * NV * gridDim.x;
        cta_sums<MMA_NT, NV>(acc, sred, part + blockIdx.x, gridDim.x);
        if (!grid_sync(A.bar, arrivals)) return false;
        grid_totals<MMA_NT>(part, nv, stot);
        slot ^= 1;
        return true;
    };
    // GenSub (MMA.cc:510-637; RobustAsymptotesType 0, no constraint
    // modification), and the older designs moved on
    double acc[NV];
#pragma unroll
    for (int j = 0; j < NV; j++) acc[j] = 0.0;
    {
        const double init = S->asyminit, dec = S->asymdec, inc = S->asyminc, feps = 1.0e-6;
        const MMAVecs &v = A.v;
        for (long long i = t0; i < n; i += ts) {
            const double x = A.x[i], lo = A.xmin[i], hi = A.xmax[i], df = A.dfdx[i], x1 = v.xo1[i];
            double Li, Ui;
            if (A.k < 3) {
                Li = x - init * (hi - lo);
                Ui = x + init * (hi - lo);
            } else {
                Li = v.L[i];
                Ui = v.U[i];
                const double helpvar = (x - x1) * (x1 - v.xo2[i]);
                const double gamma = helpvar < 0.0 ? dec : (helpvar > 0.0 ? inc : 1.0);
                Li = x - gamma * (x1 - Li);
                Ui = x + gamma * (Ui - x1);
                const double xmi = fmax(1.0e-5, hi - lo);
                Li = fmax(Li, x - 10.0 * xmi);
                Li = fmin(Li, x - 0.01 * xmi);
                Ui = fmax(Ui, x + 0.01 * xmi);
                Ui = fmin(Ui, x + 10.0 * xmi);
            }
            const double alf = fmax(lo, 0.9 * Li + 0.1 * x), bet = fmin(hi, 0.9 * Ui + 0.1 * x);
            const double ux = Ui - x, xl = x - Li, w = Ui - Li, rw = 1.0 / w;
            const double base = 0.001 * fabs(df) + 0.5 * feps * rw;
            v.xo2[i] = x1;
            v.xo1[i] = x;
            v.L[i] = Li;
            v.U[i] = Ui;
            v.p0[i] = ux * ux * (fmax(0.0, df) + base);
            v.q0[i] = xl * xl * (fmax(0.0, -df) + base);
            v.w[i] = w;
            v.rw[i] = rw;
            const double al = alf - Li, be = bet - Li, ua = Ui - alf, ub = Ui - bet;
            const double ra = 1.0 / (al * ua), rb = 1.0 / (be * ub);
            v.al[i] = al;
            v.be[i] = be;
#pragma unroll
            for (int j = 0; j < M; j++) {
                const double g = A.dgdx[(long long)j * n + i], gp = fmax(0.0, g), gm = fmax(0.0, -g);
                const double pv = ux * ux * gp, qv = xl * xl * gm;
                v.pij[(long long)j * n + i] = pv;
                v.qij[(long long)j * n + i] = qv;
                v.ga[(long long)j * n + i] = (pv * al + qv * ua) * ra;
                v.gb[(long long)j * n + i] = (pv * be + qv * ub) * rb;
                acc[j] += ux * gp + xl * gm;  // pij / (U - x) + qij / (x - L)
            }
        }
    }
    if (!reduce(acc, M)) return;
    if (threadIdx.x == 0) {  // SolveDIP initialisation (MMA.cc:642-650)
        for (int j = 0; j < M; j++) {
            D.b[j] = stot[j] - A.gx[j];
            D.lam[j] = S->c[j] / 2.0;
            D.mu[j] = 1.0;
        }
        D.epsi = 1.0;
        D.err = 1.0;
        mma_yz(D, S);
    }
    __syncthreads();
    // SolveDIP loop structure (MMA.cc:651-674): the sums at the new lambda give
    // the residual of this Newton step and the gradient and Hessian of the next
    bool bad = false;
    int loop = 0;
    for (bool first = true;; first = false) {
        double lam[M];
#pragma unroll
        for (int j = 0; j < M; j++) lam[j] = D.lam[j];
        mma_sums<M>(A, lam, acc);
        if (!reduce(acc, NV)) return;
        if (threadIdx.x == 0) {
            for (int j = 0; j < M; j++) D.G[j] = stot[j];
            int o = M;
            for (int a = 0; a < M; a++)
                for (int b = a; b < M; b++) D.H[a * M + b] = D.H[b * M + a] = stot[o++];
            if (!first) D.err = mma_residual(D, S);
            // the next epsilon that asks for a step
            while (isfinite(D.err) && D.epsi > A.tol && !(D.err > 0.9 * D.epsi && loop < 100)) {
                D.epsi = D.epsi * 0.1;
                loop = 0;
            }
            D.go = isfinite(D.err) && D.epsi > A.tol;
            if (D.go) {
                loop++;
                mma_newton(D, S);
            }
        }
        __syncthreads();
        bad = !isfinite(D.err);
        if (!D.go) break;
    }
    // x of lambda (MMA.cc:704-716)
    {
        double lam[M];
#pragma unroll
        for (int j = 0; j < M; j++) lam[j] = D.lam[j];
        for (long long i = t0; i < n; i += ts) {
            double p = A.v.p0[i], q = A.v.q0[i];
#pragma unroll
            for (int j = 0; j < M; j++) {
                p += A.v.pij[(long long)j * n + i] * lam[j];
                q += A.v.qij[(long long)j * n + i] * lam[j];
            }
            const double sp = sqrt(p), sq = sqrt(q), Li = A.v.L[i], Ui = A.v.U[i], xv = A.v.xo1[i];
            double x = (sp * Li + sq * Ui) / (sp + sq);
            const double alf = fmax(A.xmin[i], 0.9 * Li + 0.1 * xv), bet = fmin(A.xmax[i], 0.9 * Ui + 0.1 * xv);
            if (x < alf) x = alf;
            if (x > bet) x = bet;
            A.x[i] = x;
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {  // every CTA has read the scalars: all have passed the last barrier
        MMAScalars *W = A.S;
        for (int j = 0; j < M; j++) {
            W->b[j] = D.b[j];
            W->y[j] = D.y[j];
            W->lam[j] = D.lam[j];
            W->mu[j] = D.mu[j];
        }
        W->z = D.z;
        W->epsi = D.epsi;
        W->err = D.err;
    }
    if (grid_leave(A.bar)) {
        *A.status = bad ? TOPO_ERR_NAN : TOPO_OK;
        __threadfence_system();
    }
}

__global__ void k_mma_movelimit(long long n, double Xmin, double Xmax, double movlim, const double *__restrict__ x,
                                double *xmin, double *xmax) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        xmax[i] = fmin(Xmax, x[i] + movlim);
        xmin[i] = fmax(Xmin, x[i] - movlim);
    }
}

// max |x - xold| and xold <- x: the magnitudes of doubles order like their bit
// patterns, so the maximum runs on the integer pipes, one atomic per CTA
__global__ void k_mma_change(long long n, const double *__restrict__ x, double *xold, unsigned long long *bits) {
    __shared__ unsigned long long sm[EW / 32];
    unsigned long long ch = 0ull;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const double xv = x[i], d = xv - xold[i];
        const unsigned long long b = (unsigned long long)__double_as_longlong(d) & 0x7FFFFFFFFFFFFFFFull;
        if (b <= 0x7FF0000000000000ull && b > ch) ch = b;  // a NaN is passed over, as by fmax
        xold[i] = xv;
    }
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long t = __shfl_xor_sync(0xffffffffu, ch, o);
        ch = t > ch ? t : ch;
    }
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5] = ch;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < EW / 32; w++) ch = sm[w] > ch ? sm[w] : ch;
        atomicMax(bits, ch);
    }
}

// KKTresidual (MMA.cc:416-484): sums and maxima over elements
__global__ void k_mma_kkt(long long n, int m, const double *__restrict__ x, const double *__restrict__ dfdx,
                          const double *__restrict__ dgdx, const double *__restrict__ xmin,
                          const double *__restrict__ xmax, const MMAScalars *S, Partials<1> part,
                          unsigned long long *bits, double *n2out) {
    double v[1] = {0.0}, ninf = 0.0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        double ri = dfdx[i];
        for (int j = 0; j < m; j++) ri += S->lam[j] * dgdx[(long long)j * n + i];
        double mu_min = (x[i] < xmin[i] + 1.0e-5 && ri > 0.0) ? ri : 0.0;
        double mu_max = (x[i] > xmax[i] - 1.0e-5 && ri < 0.0) ? -ri : 0.0;
        ri += -mu_min + mu_max;
        double r2 = mu_min * (x[i] - xmin[i]), r3 = mu_max * (xmax[i] - x[i]);
        v[0] += ri * ri + r2 * r2 + r3 * r3;
        ninf = fmax(ninf, fmax(fabs(ri), fmax(fabs(r2), fabs(r3))));
    }
    for (int o = 16; o > 0; o >>= 1) ninf = fmax(ninf, __shfl_xor_sync(0xffffffffu, ninf, o));
    if ((threadIdx.x & 31) == 0) atomicMax(bits, (unsigned long long)__double_as_longlong(ninf));
    double tot[1];
    if (grid_reduce<EW, 1>(v, part, tot)) *n2out = tot[0];
}

// ---------------------------------------------------------------------------
int mma_create(TopoMMA **out, int n, int m, const double *a, const double *c, const double *d) {
    *out = nullptr;
    if (n < 1 || m < 1 || m > 2) {
        set_error("MMA: n >= 1 and 1 <= m <= 2 supported");
        return TOPO_ERR_ARG;
    }
    TopoMMA *mm = new TopoMMA();
    mm->n = n;
    mm->m = m;
    if (cudaStreamCreateWithFlags(&mm->stream, cudaStreamNonBlocking) != cudaSuccess) {
        delete mm;
        set_error("MMA: stream creation failed");
        return TOPO_ERR_CUDA;
    }
    auto get = [&](void **p, size_t b) -> int {
        if (cudaMalloc(p, b) != cudaSuccess) {
            cudaGetLastError();
            return TOPO_ERR_OOM;
        }
        cudaMemset(*p, 0, b);
        mm->ptrs.push_back(*p);
        return 0;
    };
    int rc = 0;
    size_t vb = sizeof(double) * (size_t)n;
    MMAVecs &v = mm->v;
    for (double **q : {&v.L, &v.U, &v.p0, &v.q0, &v.w, &v.rw, &v.al, &v.be, &v.xo1, &v.xo2}) rc |= get((void **)q, vb);
    for (double **q : {&v.pij, &v.qij, &v.ga, &v.gb}) rc |= get((void **)q, vb * m);
    rc |= get((void **)&mm->S, sizeof(MMAScalars));
    rc |= get((void **)&mm->part, sizeof(double) * 8 * 65536);
    rc |= get((void **)&mm->counter, sizeof(unsigned int) * 4);
    rc |= get((void **)&mm->bits, sizeof(unsigned long long) * 2);
    if (rc) {
        set_error("MMA: device allocation failed");
        mma_destroy(mm);
        return TOPO_ERR_OOM;
    }
    {
        const void *fn = m == 1 ? (const void *)k_mma_update<1> : (const void *)k_mma_update<2>;
        int dev = 0, nsm = 0, per_sm = 0;
        cudaError_t e = cudaHostAlloc((void **)&mm->status, sizeof(int), cudaHostAllocMapped);
        if (e == cudaSuccess) e = cudaHostGetDevicePointer((void **)&mm->status_dev, mm->status, 0);
        if (e == cudaSuccess) e = cudaGetDevice(&dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, fn, MMA_NT, 0);
        if (e != cudaSuccess || per_sm < 1) {
            set_error(std::string("MMA setup: ") + cudaGetErrorString(e));
            mma_destroy(mm);
            return TOPO_ERR_CUDA;
        }
        mm->grid = (unsigned)std::min((long long)per_sm * nsm, ((long long)n + MMA_NT - 1) / MMA_NT);
    }
    // MMA::MMA(n, m, x, a, c, d), MMA.cc:180-229
    MMAScalars &h = mm->host;
    memset(&h, 0, sizeof(h));
    h.m = m;
    h.k = 0;
    h.asyminit = 0.5;
    h.asymdec = 0.7;
    h.asyminc = 1.2;
    for (int j = 0; j < m; j++) {
        h.a[j] = a ? a[j] : 0.0;
        h.c[j] = c ? c[j] : 1000.0;
        h.d[j] = d ? d[j] : 0.0;
    }
    if (cudaMemcpy(mm->S, &h, sizeof(h), cudaMemcpyHostToDevice) != cudaSuccess) {
        set_error("MMA: upload failed");
        mma_destroy(mm);
        return TOPO_ERR_CUDA;
    }
    *out = mm;
    return TOPO_OK;
}

void mma_destroy(TopoMMA *mm) {
    if (!mm) return;
    for (void *p : mm->ptrs) cudaFree(p);
    if (mm->status) cudaFreeHost(mm->status);
    if (mm->stream) cudaStreamDestroy(mm->stream);
    delete mm;
}

int mma_set_asymptotes(TopoMMA *mm, double init, double dec, double inc) {
    mm->host.asyminit = init;
    mm->host.asymdec = dec;
    mm->host.asyminc = inc;
    MCK(cudaMemcpyAsync(&mm->S->asyminit, &mm->host.asyminit, 3 * sizeof(double), cudaMemcpyHostToDevice,
                        mm->stream));
    MCK(cudaStreamSynchronize(mm->stream));
    return TOPO_OK;
}

int mma_movelimit_dev(TopoMMA *mm, double Xmin, double Xmax, double movlim, const double *x, double *xmin,
                      double *xmax) {
    count_launch();
    k_mma_movelimit<<<ew_blocks(mm->n), EW, 0, mm->stream>>>(mm->n, Xmin, Xmax, movlim, x, xmin, xmax);
    MCK(cudaStreamSynchronize(mm->stream));
    return TOPO_OK;
}

int mma_update_dev(TopoMMA *mm, double *xval, const double *dfdx, const double *gx, const double *dgdx,
                   const double *xmin, const double *xmax) {
    cudaStream_t s = mm->stream;
    mm->host.k += 1;
    MMAArgs A;
    memset(&A, 0, sizeof(A));
    A.n = mm->n;
    A.v = mm->v;
    A.x = xval;
    A.dfdx = dfdx;
    A.dgdx = dgdx;
    A.xmin = xmin;
    A.xmax = xmax;
    for (int j = 0; j < mm->m; j++) A.gx[j] = gx[j];
    A.S = mm->S;
    A.k = mm->host.k;
    A.tol = 1.0e-9 * sqrt((double)(mm->m + mm->n));
    A.part = mm->part;
    A.bar = GridBar{mm->counter + 1, mm->counter + 2, mm->counter + 3};
    A.status = mm->status_dev;
    *mm->status = TOPO_ERR_CUDA;
    void *args[] = {&A};
    count_launch();
    MCK(cudaLaunchCooperativeKernel(mm->m == 1 ? (const void *)k_mma_update<1> : (const void *)k_mma_update<2>,
                                    dim3(mm->grid), dim3(MMA_NT), args, 0, s));
    MCK(cudaStreamSynchronize(s));
    const int st = *(volatile int *)mm->status;
    if (st == TOPO_ERR_NAN) set_error("MMA dual solve produced a non-finite residual");
    if (st == TOPO_ERR_CUDA) {  // the grid barrier gave up
        MCK(cudaMemsetAsync(mm->counter + 1, 0, 3 * sizeof(unsigned), s));
        MCK(cudaStreamSynchronize(s));
        set_error("MMA: the update's grid barrier ran out of time");
    }
    return st;
}

int mma_design_change_dev(TopoMMA *mm, const double *x, double *xold, double *ch) {
    MCK(cudaMemsetAsync(mm->bits, 0, sizeof(unsigned long long), mm->stream));
    count_launch();
    k_mma_change<<<red_blocks(mm->n), EW, 0, mm->stream>>>(mm->n, x, xold, mm->bits);
    unsigned long long b = 0;
    MCK(cudaMemcpyAsync(&b, mm->bits, sizeof(b), cudaMemcpyDeviceToHost, mm->stream));
    MCK(cudaStreamSynchronize(mm->stream));
    double v;
    memcpy(&v, &b, sizeof(v));
    *ch = v;
    return TOPO_OK;
}

int mma_kkt_dev(TopoMMA *mm, const double *x, const double *dfdx, const double *fx, const double *dgdx,
                const double *xmin, const double *xmax, double *norm2, double *normInf) {
    cudaStream_t s = mm->stream;
    MCK(cudaMemsetAsync(mm->bits, 0, sizeof(unsigned long long), s));
    double *n2d = mm->part + 8 * 65536 - 1;
    Partials<1> p1{mm->part, mm->counter};
    count_launch();
    k_mma_kkt<<<red_blocks(mm->n), EW, 0, s>>>(mm->n, mm->m, x, dfdx, dgdx, xmin, xmax, mm->S, p1, mm->bits, n2d);
    unsigned long long b = 0;
    double n2 = 0.0;
    MMAScalars h;
    MCK(cudaMemcpyAsync(&b, mm->bits, sizeof(b), cudaMemcpyDeviceToHost, s));
    MCK(cudaMemcpyAsync(&n2, n2d, sizeof(double), cudaMemcpyDeviceToHost, s));
    MCK(cudaMemcpyAsync(&h, mm->S, sizeof(h), cudaMemcpyDeviceToHost, s));
    MCK(cudaStreamSynchronize(s));
    double ninf;
    memcpy(&ninf, &b, sizeof(ninf));
    double ri = 0.0;
    for (int j = 0; j < mm->m; j++) ri += h.lam[j] * (h.a[j] * h.z + h.y[j] - fx[j]);
    n2 += ri * ri;
    ninf = fmax(fabs(ri), ninf);
    *norm2 = sqrt(n2);
    *normInf = ninf;
    return TOPO_OK;
}

int mma_restart_set_dev(TopoMMA *mm, int itr, const double *xo1, const double *xo2, const double *U,
                        const double *L) {
    if (itr < 0) {
        set_error("MMA restart: negative iteration counter");
        return TOPO_ERR_ARG;
    }
    // the reference accepts itr < 3 with a warning ("NOT A LEGAL RESTART POINT")
    const size_t b = sizeof(double) * (size_t)mm->n;
    cudaStream_t s = mm->stream;
    MCK(cudaMemcpyAsync(mm->v.xo1, xo1, b, cudaMemcpyDeviceToDevice, s));
    MCK(cudaMemcpyAsync(mm->v.xo2, xo2, b, cudaMemcpyDeviceToDevice, s));
    MCK(cudaMemcpyAsync(mm->v.U, U, b, cudaMemcpyDeviceToDevice, s));
    MCK(cudaMemcpyAsync(mm->v.L, L, b, cudaMemcpyDeviceToDevice, s));
    mm->host.k = itr;
    MCK(cudaStreamSynchronize(s));
    return TOPO_OK;
}

int mma_restart_get_dev(TopoMMA *mm, double *xo1, double *xo2, double *U, double *L) {
    const size_t b = sizeof(double) * (size_t)mm->n;
    cudaStream_t s = mm->stream;
    MCK(cudaMemcpyAsync(xo1, mm->v.xo1, b, cudaMemcpyDeviceToDevice, s));
    MCK(cudaMemcpyAsync(xo2, mm->v.xo2, b, cudaMemcpyDeviceToDevice, s));
    MCK(cudaMemcpyAsync(U, mm->v.U, b, cudaMemcpyDeviceToDevice, s));
    MCK(cudaMemcpyAsync(L, mm->v.L, b, cudaMemcpyDeviceToDevice, s));
    MCK(cudaStreamSynchronize(s));
    return TOPO_OK;
}

int mma_n(const TopoMMA *mm) { return mm->n; }
int mma_m(const TopoMMA *mm) { return mm->m; }
void *mma_stream(TopoMMA *mm) { return mm->stream; }

}  // namespace topo
