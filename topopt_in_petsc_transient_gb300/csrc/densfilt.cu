// densfilt.cu -- Filter for filterType 0 (sensitivity filter) and 1 (density
// filter), Filter.cc:60-206 and :302-531, on the element grid.
//
// H has entries R - dist between element centres for dist < R inside a box
// stencil: half-width ElemConn = max_a(ceil(R/h_a) - 1) (at least 1), the
// range along axis a running from max(i - ElemConn, 0) to
// min(i + ElemConn, n_a - 1, i + ceil(R/h_a) - 1) (Filter.cc:467-469); with
// ElemConn == 1 H is the identity (:451-459).  Hs = H 1.  The reference
// assembles H as a sparse matrix; here the weights depend only on the element
// offset and are symmetric in each axis, so one table of (ElemConn + 1)^3
// weights and one stencil kernel apply H on the fly.
//   filter 1: xTilde = (H x) ./ Hs;  dfdx, dgdx <- H (v ./ Hs)
//   filter 0: xTilde = x;           dfdx <- ((H (dfdx .* x)) ./ Hs) ./ x
// followed / preceded by the smoothed Heaviside projection and its chain rule
// (Filter.h:80-88).
#include <cmath>
#include <string>
#include <vector>

#include "kernels.cuh"
#include "le.h"
#include "planes.cuh"

namespace topo {

struct TopoDensFilt {
    int ex = 0, ey = 0, ez = 0, ftype = 1, sw = 1;
    int lim[3] = {0, 0, 0};  // upper offsets along x, y, z: min(sw, ceil(R/h_a) - 1)
    bool identity = true;
    int nsm = 1;
    long long nel = 0;
    double *w = nullptr;    // (2 sw + 1)^3 weights, offsets (dz, dy, dx) with dx fastest
    std::vector<double> wh; // the same on the host
    double *hs = nullptr;   // row sums of H
    double *tmp = nullptr;  // the scaled inputs of up to DENS_COLS columns
    double *part = nullptr;           // per-CTA partial sums of the MND reduction, and its result
    unsigned int *counter = nullptr;
    cudaStream_t stream = nullptr;
};

constexpr int DENS_COLS = 2;  // columns filtered by one launch

// post-scaling of the sum
enum { DF_POST_NONE = 0, DF_POST_DIV_HS = 1, DF_POST_DIV_HS_X = 2 };

struct DensOut {
    double *y[DENS_COLS];
    const double *hs, *x;
    int post;
    double *xp;  // the projected (or copied) result besides (one column)
    Projection proj;
};
__device__ __forceinline__ void dens_put(const DensOut &o, int col, long long e, double acc) {
    if (o.post == DF_POST_DIV_HS) acc = acc / o.hs[e];
    else if (o.post == DF_POST_DIV_HS_X) acc = (acc / o.hs[e]) / o.x[e];
    o.y[col][e] = acc;
    if (o.xp) o.xp[e] = project(o.proj, acc);
}

// y_e = post_e(sum_{e2} w(e2 - e) v_e2), one thread an element and one FP64
// multiply-add a neighbour: the form for stencils wider than DENS_SW
static __global__ void k_dens_apply(int ex, int ey, int ez, int sw, int lx, int ly, int lz,
                                    const double *__restrict__ w, const double *__restrict__ vcol, DensOut o) {
    const long long nel = (long long)ex * ey * ez;
    const int S = 2 * sw + 1, col = blockIdx.y;
    const double *v = vcol + col * nel;
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < nel; e += (long long)gridDim.x * blockDim.x) {
        int i, j, k;
        lex3(e, ex, ey, i, j, k);
        const int k0 = -min(sw, k), k1 = min(lz, ez - 1 - k);
        const int j0 = -min(sw, j), j1 = min(ly, ey - 1 - j);
        const int i0 = -min(sw, i), i1 = min(lx, ex - 1 - i);
        double acc = 0.0;
        for (int dk = k0; dk <= k1; dk++)
            for (int dj = j0; dj <= j1; dj++) {
                const double *wr = w + ((dk + sw) * S + (dj + sw)) * S + sw;
                const long long row = (long long)ex * ((j + dj) + (long long)ey * (k + dk)) + i;
                for (int di = i0; di <= i1; di++) {
                    const double wt = wr[di];
                    if (wt == 0.0) continue;
                    acc += wt * v[row + di];
                }
            }
        dens_put(o, col, e, acc);
    }
}

// The same for half-widths up to DENS_SW, by symmetry: with t_a the sum of the
// values at distance a along x, s_ab that of t_a at distance b along y, and
// G_c = sum_ab w_abc s_ab in a plane, the result adds G_c of the planes at
// distance c.  Marched along z, a column of elements per thread, the partial
// results of 2 SW + 1 planes in registers.  FP64 instructions an element bound
// it (GB300: 2 lanes a clock and SM): 34 and an eighth-odd rim for SW = 2 and R =
// 3 against 93 neighbours, each with a quotient before the inputs were scaled
// ahead of the sums: filter and chain rule of three fields take 0.25 ms at
// 96x48x48 and R = 3 instead of 1.45.
constexpr int DENS_SW = 4;
constexpr int DN_T = 256, DN_SLOTS = 4;
template <int SW>
struct DensW {
    double w[(SW + 1) * (SW + 1) * (SW + 1)];  // [c][b][a]
};
template <int SW>
static __global__ void __launch_bounds__(DN_T, 2)
    k_dens_march(int ex, int ey, int ez, Patch P, int cz, const DensW<SW> W, const double *__restrict__ vcol, DensOut o) {
    TOPO_DYNAMIC_SMEM(double, sm);
    constexpr int A1 = SW + 1;
    const int tid = threadIdx.x, ly = tid / P.tx, lx = tid - ly * P.tx, col = blockIdx.y;
    const int row = P.tx + 2 * SW, rows = P.ty + 2 * SW, nst = row * rows, nt = P.tx * rows;
    double *raw = sm, *t = sm + nst;  // staged plane; x sums [a][rows][tx]
    int b = blockIdx.x;
    const int bx = b % P.ntx;
    b /= P.ntx;
    const int i0 = bx * P.tx, j0 = (b % P.nty) * P.ty, k0 = (b / P.nty) * cz, k1 = min(k0 + cz, ez);
    const int i = i0 + lx, j = j0 + ly;
    const bool in = ly < P.ty && i < ex && j < ey;
    const long long nxy = (long long)ex * ey;
    const double *v = vcol + col * nxy * ez;
    int sn[DN_SLOTS];  // staged elements of this thread within a plane (-1: outside the domain)
#pragma unroll
    for (int q = 0; q < DN_SLOTS; q++) {
        const int s = tid + q * DN_T, r = s / row, si = i0 - SW + s - r * row, sj = j0 - SW + r;
        sn[q] = s < nst && si >= 0 && si < ex && sj >= 0 && sj < ey ? si + ex * sj : -1;
    }
    double reg[DN_SLOTS], acc[2 * SW + 1];
    auto fetch = [&](int k) {
#pragma unroll
        for (int q = 0; q < DN_SLOTS; q++) reg[q] = k >= 0 && k < ez && sn[q] >= 0 ? v[sn[q] + nxy * k] : 0.0;
    };
#pragma unroll
    for (int q = 0; q < 2 * SW + 1; q++) acc[q] = 0.0;
    fetch(k0 - SW);
    for (int p = k0 - SW; p < k1 + SW; p++) {  // acc[q]: result of plane p - SW + q
#pragma unroll
        for (int q = 0; q < DN_SLOTS; q++)
            if (tid + q * DN_T < nst) raw[tid + q * DN_T] = reg[q];
        __syncthreads();
        fetch(p + 1);
        for (int s = tid; s < nt; s += DN_T) {
            const int r = s / P.tx, x = s - r * P.tx;
            const double *c = raw + r * row + x + SW;
            t[s] = c[0];
#pragma unroll
            for (int a = 1; a <= SW; a++) t[a * nt + s] = c[-a] + c[a];
        }
        __syncthreads();
        if (in) {
            double G[A1];
#pragma unroll
            for (int c = 0; c <= SW; c++) G[c] = 0.0;
#pragma unroll
            for (int a = 0; a <= SW; a++)
#pragma unroll
                for (int bb = 0; bb <= SW; bb++) {
                    if (W.w[bb * A1 + a] == 0.0) continue;  // no weight in any plane: the same in every thread
                    const double *c = t + a * nt + (ly + SW) * P.tx + lx;
                    const double s = bb ? c[-bb * P.tx] + c[bb * P.tx] : c[0];
#pragma unroll
                    for (int c2 = 0; c2 <= SW; c2++)
                        if (W.w[(c2 * A1 + bb) * A1 + a] != 0.0) G[c2] += W.w[(c2 * A1 + bb) * A1 + a] * s;
                }
#pragma unroll
            for (int q = 0; q < 2 * SW + 1; q++) acc[q] += G[q < SW ? SW - q : q - SW];
            if (p - SW >= k0) dens_put(o, col, i + (long long)ex * j + nxy * (p - SW), acc[0]);
#pragma unroll
            for (int q = 0; q < 2 * SW; q++) acc[q] = acc[q + 1];
            acc[2 * SW] = 0.0;
        }
        // the next plane's values go to raw, read last before the barrier above; t is rewritten after the next one
    }
}

// inputs of the sums, column c of `cols`: the chain rule of the projection
// (Filter.cc:128-169) on dfdx (c = 0) and dgdx, then the pre-scaling: x
// (sensitivity filter, dfdx alone; dgdx takes the chain rule in place) or 1 / Hs
static __global__ void k_dens_pre(long long nel, const double *__restrict__ xt, const double *__restrict__ x,
                                  const double *__restrict__ hs, double *c0, double *c1, double *t0, double *t1,
                                  Projection pr) {
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < nel; e += (long long)gridDim.x * blockDim.x) {
        const double d = pr.on ? project_slope(pr, xt[e]) : 1.0;
        double v0 = c0[e], v1 = c1 ? c1[e] : 0.0;
        if (pr.on) {
            v0 *= d;
            v1 *= d;
        }
        if (x) {  // sensitivity filter
            t0[e] = v0 * x[e];
            if (c1 && pr.on) c1[e] = v1;
        } else {
            const double h = hs[e];
            t0[e] = v0 / h;
            if (c1) t1[e] = v1 / h;
        }
    }
}

// Filter::GetMND (Filter.cc:208-227): mean of 4 x (1 - x)
static __global__ void k_dens_mnd(long long n, const double *__restrict__ x, Partials<1> part, double *out) {
    double v[1] = {0.0};
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x)
        v[0] += 4 * x[e] * (1.0 - x[e]);
    double tot[1];
    if (grid_reduce<EW, 1>(v, part, tot)) *out = tot[0] / (double)n;
}

static __global__ void k_dens_fill(long long n, double v, double *y) {
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < n; e += (long long)gridDim.x * blockDim.x)
        y[e] = v;
}

// xTilde = v and xPhys from it: smoothed Heaviside projection or copy
// (Filter.cc:110-116); identity H and the sensitivity filter
static __global__ void k_dens_project(long long nel, const double *__restrict__ v, double *xt, double *xp,
                                      Projection pr) {
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < nel; e += (long long)gridDim.x * blockDim.x) {
        const double x = v[e];
        xt[e] = x;
        xp[e] = project(pr, x);
    }
}

// identity H: the chain rule of the projection (Filter.cc:128-169) on one column;
// the filter's own scalings by Hs = 1 and by x and 1 / x cancel up to rounding,
// which is kept: (v x) / x
static __global__ void k_dens_identity(long long nel, const double *__restrict__ xt, const double *__restrict__ x,
                                       double *v, Projection pr) {
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < nel; e += (long long)gridDim.x * blockDim.x) {
        double a = v[e];
        if (pr.on) a *= project_slope(pr, xt[e]);
        if (x) a = (a * x[e]) / x[e];
        v[e] = a;
    }
}

#define DCK(call)                                                            \
    do {                                                                     \
        cudaError_t e_ = (call);                                             \
        if (e_ != cudaSuccess) {                                             \
            set_error(std::string(#call) + ": " + cudaGetErrorString(e_));  \
            return TOPO_ERR_CUDA;                                            \
        }                                                                    \
    } while (0)

// H on the ncol columns at v, post-scaled into o
template <int SW>
static void dens_march(TopoDensFilt *f, const double *v, int ncol, const DensOut &o) {
    DensW<SW> W;
    const int S = 2 * SW + 1;
    for (int c = 0; c <= SW; c++)
        for (int b = 0; b <= SW; b++)
            for (int a = 0; a <= SW; a++)
                W.w[(c * (SW + 1) + b) * (SW + 1) + a] = f->wh[((size_t)(c + SW) * S + (b + SW)) * S + (a + SW)];
    const Patch P = plane_patch(f->ex, f->ey, DN_T, SW, DN_SLOTS * DN_T);
    // runs of planes: the fewest plane steps of the busiest SM, a run taking 2 SW more than it completes
    int best = f->ez;
    double bt = 1e300;
    for (int nz = 1; nz <= f->ez; nz++) {
        const int cz = (f->ez + nz - 1) / nz;
        const long long ctas = (long long)P.ntx * P.nty * ((f->ez + cz - 1) / cz) * ncol;
        const double t = (double)((ctas + f->nsm - 1) / f->nsm) * (cz + 2 * SW);
        if (t < bt) {
            bt = t;
            best = cz;
        }
    }
    const size_t sm = sizeof(double) * ((size_t)(P.tx + 2 * SW) * (P.ty + 2 * SW) +
                                        (size_t)(SW + 1) * P.tx * (P.ty + 2 * SW));  // at most 41 KB
    const dim3 grid((unsigned)(P.ntx * P.nty * ((f->ez + best - 1) / best)), (unsigned)ncol);
    k_dens_march<SW><<<grid, DN_T, sm, f->stream>>>(f->ex, f->ey, f->ez, P, best, W, v, o);
}
static void dens_apply(TopoDensFilt *f, const double *v, int ncol, const DensOut &o) {
    count_launch();
    if (f->sw == 2) dens_march<2>(f, v, ncol, o);
    else if (f->sw == 3) dens_march<3>(f, v, ncol, o);
    else if (f->sw == DENS_SW) dens_march<DENS_SW>(f, v, ncol, o);
    else
        k_dens_apply<<<dim3(ew_blocks(f->nel), (unsigned)ncol), EW, 0, f->stream>>>(
            f->ex, f->ey, f->ez, f->sw, f->lim[0], f->lim[1], f->lim[2], f->w, v, o);
}

static void dens_destroy(TopoDensFilt *f) {
    if (!f) return;
    cudaFree(f->w);
    cudaFree(f->hs);
    cudaFree(f->tmp);
    cudaFree(f->part);
    cudaFree(f->counter);
    if (f->stream) cudaStreamDestroy(f->stream);
    delete f;
}

static int dens_create(TopoDensFilt **out, int ex, int ey, int ez, double hx, double hy, double hz, int ftype,
                       double R) {
    *out = nullptr;
    if (ex < 1 || ey < 1 || ez < 1 || hx <= 0.0 || hy <= 0.0 || hz <= 0.0 || !(R > 0.0) || (ftype != 0 && ftype != 1)) {
        set_error("Filter: filter type 0 or 1, positive element sizes and radius");
        return TOPO_ERR_ARG;
    }
    TopoDensFilt *f = new TopoDensFilt();
    f->ex = ex;
    f->ey = ey;
    f->ez = ez;
    f->ftype = ftype;
    f->nel = (long long)ex * ey * ez;
    const double h[3] = {hx, hy, hz};
    int sw = 0;
    for (int a = 0; a < 3; a++) {
        f->lim[a] = (int)std::ceil(R / h[a]) - 1;
        sw = std::max(sw, f->lim[a]);
    }
    if (sw == 0) sw = 1;  // Filter.cc:396-398
    f->sw = sw;
    f->identity = (sw == 1);  // Filter.cc:451-459
    for (int a = 0; a < 3; a++) f->lim[a] = std::min(f->lim[a], sw);
    const int S = 2 * sw + 1;
    std::vector<double> w((size_t)S * S * S, 0.0);
    for (int dk = -sw; dk <= sw; dk++)
        for (int dj = -sw; dj <= sw; dj++)
            for (int di = -sw; di <= sw; di++) {
                // element centres h/2 + i h (DMDASetUniformCoordinates, Filter.cc:420)
                const double d0 = (hx / 2 + di * hx) - hx / 2, d1 = (hy / 2 + dj * hy) - hy / 2,
                             d2 = (hz / 2 + dk * hz) - hz / 2;
                const double dist = std::sqrt(d0 * d0 + d1 * d1 + d2 * d2);
                w[((size_t)(dk + sw) * S + (dj + sw)) * S + (di + sw)] = dist < R ? R - dist : 0.0;
            }
    f->wh = w;
    int dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&f->nsm, cudaDevAttrMultiProcessorCount, dev);
    f->nsm = std::max(f->nsm, 1);
    bool ok = cudaStreamCreateWithFlags(&f->stream, cudaStreamNonBlocking) == cudaSuccess &&
              cudaMalloc(&f->w, sizeof(double) * w.size()) == cudaSuccess &&
              cudaMalloc(&f->hs, sizeof(double) * f->nel) == cudaSuccess &&
              cudaMalloc(&f->tmp, sizeof(double) * DENS_COLS * f->nel) == cudaSuccess &&
              cudaMalloc(&f->part, sizeof(double) * (red_blocks(f->nel) + 1)) == cudaSuccess &&
              cudaMalloc(&f->counter, sizeof(unsigned int)) == cudaSuccess &&
              cudaMemset(f->counter, 0, sizeof(unsigned int)) == cudaSuccess;
    if (!ok) {
        cudaGetLastError();
        dens_destroy(f);
        set_error("Filter: device allocation failed");
        return TOPO_ERR_OOM;
    }
    cudaError_t e = cudaMemcpy(f->w, w.data(), sizeof(double) * w.size(), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        count_launch();
        k_dens_fill<<<ew_blocks(f->nel), EW, 0, f->stream>>>(f->nel, 1.0, f->identity ? f->hs : f->tmp);
        // Hs = H 1 (Filter.cc:505-509) by the sums that it divides: a solid density stays 1
        // exactly, and rounding that both share cancels (against 80 bits, R = 3: xTilde
        // 1.7e-16 instead of 9.3e-16 with Hs summed in the reference's column order)
        if (!f->identity) {
            DensOut o{};
            o.y[0] = f->hs;
            dens_apply(f, f->tmp, 1, o);
        }
        e = cudaStreamSynchronize(f->stream);
    }
    if (e != cudaSuccess) {
        set_error(std::string("Filter set-up: ") + cudaGetErrorString(e));
        dens_destroy(f);
        return TOPO_ERR_CUDA;
    }
    *out = f;
    return TOPO_OK;
}

static int dens_project_dev(TopoDensFilt *f, const double *x, double *xt, double *xp, int projection, double beta,
                            double eta) {
    const Projection pr = make_projection(projection, beta, eta);
    if (f->ftype == 1 && !f->identity) {
        DensOut o{};
        o.y[0] = xt;
        o.hs = f->hs;
        o.post = DF_POST_DIV_HS;
        o.xp = xp;
        o.proj = pr;
        // the sums read neighbours: a result written over its input needs a copy of it
        const double *v = x;
        if (x == xt || x == xp) {
            DCK(cudaMemcpyAsync(f->tmp, x, sizeof(double) * f->nel, cudaMemcpyDeviceToDevice, f->stream));
            v = f->tmp;
        }
        dens_apply(f, v, 1, o);
    } else {
        count_launch();
        k_dens_project<<<ew_blocks(f->nel), EW, 0, f->stream>>>(f->nel, x, xt, xp, pr);
    }
    DCK(cudaGetLastError());
    DCK(cudaStreamSynchronize(f->stream));
    return TOPO_OK;
}

static int dens_gradients_dev(TopoDensFilt *f, const double *x, const double *xt, double *df, int m, double *dg,
                              int projection, double beta, double eta) {
    const long long nel = f->nel;
    const unsigned nb = ew_blocks(nel);
    const Projection pr = make_projection(projection, beta, eta);
    for (int j = -1; j < m; j += DENS_COLS) {  // column -1: dfdx (Filter.cc:172-195)
        double *c0 = j < 0 ? df : dg + (size_t)j * nel, *c1 = j + 1 < m ? dg + (size_t)(j + 1) * nel : nullptr;
        // the sensitivity filter leaves dgdx to the chain rule
        const bool filt0 = f->ftype == 1 || j < 0, filt1 = c1 && f->ftype == 1;
        if (f->identity || !filt0) {
            if (projection || (f->ftype == 0 && j < 0)) {
                count_launch();
                k_dens_identity<<<nb, EW, 0, f->stream>>>(nel, xt, f->ftype == 0 && j < 0 ? x : nullptr, c0, pr);
            }
            if (c1 && projection) {
                count_launch();
                k_dens_identity<<<nb, EW, 0, f->stream>>>(nel, xt, nullptr, c1, pr);
            }
            continue;
        }
        count_launch();
        k_dens_pre<<<nb, EW, 0, f->stream>>>(nel, xt, f->ftype == 0 ? x : nullptr, f->hs, c0, c1, f->tmp, f->tmp + nel, pr);
        DensOut o{};
        o.y[0] = c0;
        o.y[1] = c1;
        o.hs = f->hs;
        o.x = x;
        o.post = f->ftype == 0 ? DF_POST_DIV_HS_X : DF_POST_NONE;
        dens_apply(f, f->tmp, filt1 ? 2 : 1, o);
    }
    DCK(cudaGetLastError());
    DCK(cudaStreamSynchronize(f->stream));
    return TOPO_OK;
}

static int dens_mnd_dev(TopoDensFilt *f, const double *x, double *mnd) {
    const unsigned nb = red_blocks(f->nel);
    count_launch();
    k_dens_mnd<<<nb, EW, 0, f->stream>>>(f->nel, x, Partials<1>{f->part, f->counter}, f->part + nb);
    DCK(cudaMemcpyAsync(mnd, f->part + nb, sizeof(double), cudaMemcpyDeviceToHost, f->stream));
    DCK(cudaStreamSynchronize(f->stream));
    return TOPO_OK;
}

}  // namespace topo

using namespace topo;

struct topo_densfilt {
    TopoDensFilt *impl = nullptr;
    long long nel = 0;
    double *d_a = nullptr, *d_b = nullptr, *d_c = nullptr, *d_d = nullptr, *d_g = nullptr;  // host-call staging
    int gcap = 2;
};

extern "C" {

int topo_densfilt_create(topo_densfilt **out, int nelx, int nely, int nelz, double hx, double hy, double hz,
                         int filter_type, double rmin) {
    if (!out) return TOPO_ERR_ARG;
    *out = nullptr;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
        cudaGetLastError();
        set_error("no CUDA device available: the GB300 path has no CPU fallback");
        return TOPO_ERR_CUDA;
    }
    TopoDensFilt *impl = nullptr;
    int rc = dens_create(&impl, nelx, nely, nelz, hx, hy, hz, filter_type, rmin);
    if (rc) return rc;
    topo_densfilt *h = new topo_densfilt();
    h->impl = impl;
    h->nel = impl->nel;
    const size_t b = sizeof(double) * h->nel;
    bool ok = cudaMalloc(&h->d_a, b) == cudaSuccess && cudaMalloc(&h->d_b, b) == cudaSuccess &&
              cudaMalloc(&h->d_c, b) == cudaSuccess && cudaMalloc(&h->d_d, b) == cudaSuccess &&
              cudaMalloc(&h->d_g, b * h->gcap) == cudaSuccess;
    if (!ok) {
        cudaGetLastError();
        topo_densfilt_destroy(h);
        set_error("device allocation of Filter staging buffers failed");
        return TOPO_ERR_OOM;
    }
    *out = h;
    return TOPO_OK;
}

void topo_densfilt_destroy(topo_densfilt *f) {
    if (!f) return;
    dens_destroy(f->impl);
    cudaFree(f->d_a);
    cudaFree(f->d_b);
    cudaFree(f->d_c);
    cudaFree(f->d_d);
    cudaFree(f->d_g);
    delete f;
}

int topo_densfilt_filter_project_dev(topo_densfilt *f, const double *x_dev, double *xTilde_dev, double *xPhys_dev,
                                     int projection, double beta, double eta) {
    if (!f || !x_dev || !xTilde_dev || !xPhys_dev) return TOPO_ERR_ARG;
    return dens_project_dev(f->impl, x_dev, xTilde_dev, xPhys_dev, projection, beta, eta);
}

int topo_densfilt_filter_project(topo_densfilt *f, const double *x, double *xTilde, double *xPhys, int projection,
                                 double beta, double eta) {
    if (!f || !x || !xTilde || !xPhys) return TOPO_ERR_ARG;
    const size_t b = sizeof(double) * f->nel;
    DCK(cudaMemcpy(f->d_a, x, b, cudaMemcpyHostToDevice));
    int rc = dens_project_dev(f->impl, f->d_a, f->d_b, f->d_c, projection, beta, eta);
    if (rc) return rc;
    DCK(cudaMemcpy(xTilde, f->d_b, b, cudaMemcpyDeviceToHost));
    DCK(cudaMemcpy(xPhys, f->d_c, b, cudaMemcpyDeviceToHost));
    return TOPO_OK;
}

int topo_densfilt_gradients_dev(topo_densfilt *f, const double *x_dev, const double *xTilde_dev, double *dfdx_dev,
                                int m, double *dgdx_dev, int projection, double beta, double eta) {
    if (!f || !x_dev || !xTilde_dev || !dfdx_dev || m < 0 || (m > 0 && !dgdx_dev)) return TOPO_ERR_ARG;
    return dens_gradients_dev(f->impl, x_dev, xTilde_dev, dfdx_dev, m, dgdx_dev, projection, beta, eta);
}

int topo_densfilt_gradients(topo_densfilt *f, const double *x, const double *xTilde, double *dfdx, int m,
                            double *dgdx, int projection, double beta, double eta) {
    if (!f || !x || !xTilde || !dfdx || m < 0 || m > f->gcap || (m > 0 && !dgdx)) return TOPO_ERR_ARG;
    const size_t b = sizeof(double) * f->nel;
    DCK(cudaMemcpy(f->d_a, x, b, cudaMemcpyHostToDevice));
    DCK(cudaMemcpy(f->d_b, xTilde, b, cudaMemcpyHostToDevice));
    DCK(cudaMemcpy(f->d_c, dfdx, b, cudaMemcpyHostToDevice));
    if (m) DCK(cudaMemcpy(f->d_g, dgdx, b * m, cudaMemcpyHostToDevice));
    int rc = dens_gradients_dev(f->impl, f->d_a, f->d_b, f->d_c, m, f->d_g, projection, beta, eta);
    if (rc) return rc;
    DCK(cudaMemcpy(dfdx, f->d_c, b, cudaMemcpyDeviceToHost));
    if (m) DCK(cudaMemcpy(dgdx, f->d_g, b * m, cudaMemcpyDeviceToHost));
    return TOPO_OK;
}

int topo_densfilt_mnd_dev(topo_densfilt *f, const double *x_dev, double *mnd) {
    if (!f || !x_dev || !mnd) return TOPO_ERR_ARG;
    return dens_mnd_dev(f->impl, x_dev, mnd);
}

int topo_densfilt_mnd(topo_densfilt *f, const double *x, double *mnd) {
    if (!f || !x || !mnd) return TOPO_ERR_ARG;
    DCK(cudaMemcpy(f->d_a, x, sizeof(double) * f->nel, cudaMemcpyHostToDevice));
    return dens_mnd_dev(f->impl, f->d_a, mnd);
}

}  // extern "C"
