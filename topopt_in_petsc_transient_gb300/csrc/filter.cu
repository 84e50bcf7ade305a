// filter.cu -- PDEFilt (PDEFilter.cc) and the filter-type-2 branch of Filter
// (Filter.cc) on one GPU.
//
// The Helmholtz filter (-R^2 lap + 1) u = T x on the nodal grid has the same
// 8x8 element matrix for every element (R^2 * Laplacian + mass of the box,
// PDEFilter.cc:485-578); T (0.125 per element node, :580-588) and T^t are
// gathers.  The assembled operator is a sum of tensor products of the 1-D
// stiffness and mass, applied without the matrix; the solve is one cooperative
// kernel (k_filt_solve), with a second one for what FP32 corrections cannot solve
// (k_filt_cg).
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <utility>
#include <vector>

#include "coop.cuh"
#include "filtctl.cuh"
#include "filter.h"
#include "kernels.cuh"
#include "planes.cuh"

namespace topo {

#define FCK(call)                                                            \
    do {                                                                     \
        cudaError_t e_ = (call);                                             \
        if (e_ != cudaSuccess) {                                             \
            set_error(std::string(#call) + ": " + cudaGetErrorString(e_));  \
            return TOPO_ERR_CUDA;                                            \
        }                                                                    \
    } while (0)

constexpr int FT_N = 256;          // threads: node columns of a CTA, tx x ty of them
constexpr int FT_PLANE = 2 * FT_N;  // most values of a staged plane: the columns and one node around
constexpr int FT_RING = 4;          // planes whose raw values are in flight or in use
constexpr int FT_RAW = 12;          // most bytes of a node's raw values
struct FiltSmem {
    double plane[2][FT_PLANE];
    unsigned char ring[FT_RING][FT_PLANE * FT_RAW];
};
template <int NB>
__device__ __forceinline__ void filt_copy(void *dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src),
                 "n"(NB)
                 : "memory");
}

// Operator of the unit-scaled filter K / V (V the element volume).  The 1-D
// assembled mass and stiffness are h [1 4 1] / 6 and [-1 2 -1] / h inside, and
// at an end half of the same stencil on the mirrored line (v_-1 = v_1).  So
//   K / V = d A,  A the constant 27-point stencil
//   [m m m + sum_a (R / h_a)^2 k_a m_b m_c],  m = [1 4 1] / 6, k = [-1 2 -1],
// on the mirrored field, d = 1/2 per axis on which the node is at an end.  c[S]:
// A's weight of a neighbour displaced along the axes in S (bit a: axis a).
template <class T>
struct FiltOp {
    T c[8];
};

struct FiltStatus {
    int status;
    int hard, cur;  // bit r set for a right-hand side left to k_filt_cg; which u the others stand in
};

struct FiltArgs {
    GridDesc g;
    FiltOp<double> Kd;
    FiltOp<float> Kf;
    int nr;                             // right-hand sides
    const double *xin[FILT_RHS];        // element fields
    double *xout[FILT_RHS], *xphys;     // results; xphys: clamp and project (one right-hand side)
    int clamp;
    Projection proj;
    double *u[FILT_RHS][2], *b[FILT_RHS], *r[FILT_RHS];
    double *q[FILT_RHS];                // k_filt_cg: K p, in the storage of r32
    float *r32[FILT_RHS][2], *s32[FILT_RHS][2], *w32[FILT_RHS][2], *p32[FILT_RHS], *d32[FILT_RHS];
    // b and u are those of the element volume's power of two times the fields, so that
    // b.b keeps the range that it has with K and T of volume V
    double sb, sx;                      // T and T^t: an eighth times it, an eighth over it
    double tol;
    int maxit, fp64;                    // fp64: no corrections (filt_in_fp64)
    double *part;                       // [2 slots][FILT_RHS][gridDim] FP64 sums, then [2][FILT_RHS][3][gridDim] FP32 ones
    GridBar bar;
    FiltStatus *out;                    // mapped host memory
    int tx, ty, ntx, nty, cz, ncz;      // patches of tx x ty node columns, runs of cz planes
};

// A applied to a field in runs of planes along z, a column of nodes per thread.
// F supplies the field and takes the products:
//   copy(ring, v, n); T val(ring, v, s)   raw values of node n into slot v of a ring plane (asynchronous
//                                         copies); the node's value from them, s = 1 / d
//   Own own(n); put(n, d, Own, v, y)  node n: boundary factor, operands, own value, product
// In-plane neighbours come from one staged plane; of the two planes beside it
// only Q, the in-plane sum with the weights of a neighbour along z, is needed,
// kept in registers: 15 operations a node instead of 27 multiply-adds.  Bound by
// the latency of its loads (24 warps an SM), so the staged ones are issued three
// planes ahead of their use (2.68 -> 2.58 ms against two planes ahead in
// registers), into slots of shared memory that only their thread
// reads, and the node's own one plane ahead.
template <class T, class F>
__device__ __forceinline__ void filt_apply(const FiltArgs &A, const FiltOp<T> &K, FiltSmem &sm, F &f) {
    const GridDesc &g = A.g;
    const int tid = threadIdx.x, ty = tid / A.tx, tx = tid - ty * A.tx;
    const int row = A.tx + 2, nst = row * (A.ty + 2);
    const int items = A.ntx * A.nty * A.ncz;
    const unsigned nxy = (unsigned)g.nx * g.ny;  // node indices stay below 2^32 (lex3)
    // node index along an axis of n nodes, mirrored one beyond its ends
    auto mirror = [](int i, int n) { return min(max(i < 0 ? -i : (i >= n ? 2 * n - 2 - i : i), 0), n - 1); };
    for (int it = blockIdx.x; it < items; it += gridDim.x) {
        const int bx = it % A.ntx, by = (it / A.ntx) % A.nty, bz = it / (A.ntx * A.nty);
        const int i0 = bx * A.tx, j0 = by * A.ty, k0 = bz * A.cz, k1 = min(k0 + A.cz, g.nz);
        const int i = i0 + tx, j = j0 + ty;
        const bool in = ty < A.ty && i < g.nx && j < g.ny;
        const float dxy = ((i == 0 || i == g.nx - 1) ? 0.5f : 1.0f) * ((j == 0 || j == g.ny - 1) ? 0.5f : 1.0f);
        const unsigned nij = i + (unsigned)g.nx * j;
        int sn[2];    // staged nodes of this thread within a plane (-1: none) and their 1 / d
        float ss[2];
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const int v = tid + q * FT_N, r = v / row;
            const int si = mirror(i0 - 1 + v - r * row, g.nx), sj = mirror(j0 - 1 + r, g.ny);
            sn[q] = v < nst ? si + g.nx * sj : -1;
            ss[q] = ((si == 0 || si == g.nx - 1) ? 2.0f : 1.0f) * ((sj == 0 || sj == g.ny - 1) ? 2.0f : 1.0f);
        }
        typename F::Own own[2];  // of the planes k (being staged) and k - 1 (being completed)
        auto fetch = [&](int k) {  // one group of copies a plane, empty past the run
            if (k <= k1) {
                const unsigned o = nxy * (unsigned)mirror(k, g.nz);
#pragma unroll
                for (int q = 0; q < 2; q++)
                    if (sn[q] >= 0) f.copy(sm.ring[k & (FT_RING - 1)], tid + q * FT_N, o + sn[q]);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        T vc = T(0), P = T(0), Q = T(0), Ql = T(0);
        auto step = [&](int k, typename F::Own &ok, const typename F::Own &okm1) {
            T *pl = reinterpret_cast<T *>(sm.plane[k & 1]);
            asm volatile("cp.async.wait_group %0;" ::"n"(FT_RING - 2) : "memory");  // this thread's copies of plane k
            const float sz = (k <= 0 || k >= g.nz - 1) && k != -1 && k != g.nz ? 2.0f : 1.0f;
            // beyond an end the mirrored plane 1 or nz - 2 is staged, itself an end plane when nz = 2
            const float s2 = (k == -1 || k == g.nz) && g.nz == 2 ? 2.0f : sz;
#pragma unroll
            for (int q = 0; q < 2; q++)
                if (sn[q] >= 0) pl[tid + q * FT_N] = f.val(sm.ring[k & (FT_RING - 1)], tid + q * FT_N, s2 * ss[q]);
            fetch(k + FT_RING - 1);
            if (in && k >= k0 && k < k1) ok = f.own(nij + nxy * (unsigned)k);
            __syncthreads();  // one barrier a plane: the other buffer was last read before the previous one
            if (in) {
                const T *s = pl + (ty + 1) * row + tx + 1, *su = s + row, *sd = s - row;
                const T c = s[0], ax = s[-1] + s[1], ay = su[0] + sd[0], axy = (su[-1] + su[1]) + (sd[-1] + sd[1]);
                const T Qn = K.c[4] * c + K.c[5] * ax + K.c[6] * ay + K.c[7] * axy;
                if (k > k0)  // plane k - 1 is complete
                    f.put(nij + nxy * (unsigned)(k - 1), (k == 1 || k == g.nz) ? 0.5f * dxy : dxy, okm1, vc,
                          P + (Ql + Qn));
                P = K.c[0] * c + K.c[1] * ax + K.c[2] * ay + K.c[3] * axy;
                Ql = Q;
                Q = Qn;
                vc = c;
            }
        };
#pragma unroll
        for (int k = 0; k < FT_RING - 1; k++) fetch(k0 - 1 + k);
        for (int k = k0 - 1; k <= k1; k += 2) {  // by two: the operands swap by name, no copies that wait for loads
            step(k, own[0], own[1]);
            if (k + 1 <= k1) step(k + 1, own[1], own[0]);
        }
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();  // the planes are restaged by the next run
    }
}

// start of a correction: r32 = r / rms(r), z = Dinv r32, w = K z, d = 0
struct FiltStart {
    const double *r64;
    ScaleF64 sg;
    float dinv, *r, *w, *d, sum[3];
    using Own = double;
    __device__ void copy(unsigned char *ring, int v, unsigned n) const { filt_copy<8>((double *)ring + v, r64 + n); }
    __device__ float val(const unsigned char *ring, int v, float s) const {
        return s * dinv * scaled_f32(((const double *)ring)[v], sg);
    }
    __device__ Own own(unsigned n) const { return r64[n]; }
    __device__ void put(unsigned n, float bd, Own v, float z, float y) {
        const float rv = scaled_f32(v, sg), wv = bd * y;
        r[n] = rv;
        w[n] = wv;
        d[n] = 0.0f;
        sum[0] += rv * z;
        sum[1] += wv * z;
    }
};
// one CG iteration (k_filt_solve)
struct FiltIter {
    float al, be, dinv;
    const float *ro, *so, *wo;
    float *rn, *sn, *wn, *p, *d, sum[3];
    struct Own {
        float r, w, s, p, d;
    };
    // beta = 0 (the first step): s and p may hold anything
    __device__ float snew(float w, float s) const { return be == 0.0f ? w : w + be * s; }
    __device__ void copy(unsigned char *ring, int v, unsigned n) const {
        float *q = (float *)ring + v;
        filt_copy<4>(q, ro + n);
        filt_copy<4>(q + FT_PLANE, wo + n);
        filt_copy<4>(q + 2 * FT_PLANE, so + n);
    }
    __device__ float val(const unsigned char *ring, int v, float s) const {
        const float *q = (const float *)ring + v;
        return s * dinv * (q[0] - al * snew(q[FT_PLANE], q[2 * FT_PLANE]));
    }
    __device__ Own own(unsigned n) const { return {ro[n], wo[n], so[n], p[n], d[n]}; }
    __device__ void put(unsigned n, float bd, const Own &o, float z, float y) {
        const float sv = snew(o.w, o.s), rv = o.r - al * sv, zold = dinv * o.r * (bd == 1.0f ? 1.0f : 1.0f / bd);
        const float pv = be == 0.0f ? zold : zold + be * o.p, wv = bd * y;
        sn[n] = sv;
        rn[n] = rv;
        p[n] = pv;
        d[n] = o.d + al * pv;
        wn[n] = wv;
        sum[0] += rv * z;
        sum[1] += wv * z;
        sum[2] += rv * rv;
    }
};
// end of a correction: u += d / sigma, r = b - K u
struct FiltResid {
    const double *uo, *b;
    const float *d;
    double is, *un, *r, sum;
    using Own = double;
    __device__ void copy(unsigned char *ring, int v, unsigned n) const {
        filt_copy<8>((double *)ring + v, uo + n);
        filt_copy<4>((float *)(ring + 8 * FT_PLANE) + v, d + n);
    }
    __device__ double val(const unsigned char *ring, int v, float) const {
        return fma(is, f32_to_f64(((const float *)(ring + 8 * FT_PLANE))[v]), ((const double *)ring)[v]);
    }
    __device__ Own own(unsigned n) const { return b[n]; }
    __device__ void put(unsigned n, float bd, Own bv, double v, double y) {
        un[n] = v;
        const double e = bv - (bd == 1.0f ? y : (double)bd * y);
        r[n] = e;
        sum += e * e;
    }
};

// K p of k_filt_cg
struct FiltMul {
    const double *p;
    double *q, sum;
    struct Own {};
    __device__ void copy(unsigned char *ring, int v, unsigned n) const { filt_copy<8>((double *)ring + v, p + n); }
    __device__ double val(const unsigned char *ring, int v, float) const { return ((const double *)ring)[v]; }
    __device__ Own own(unsigned) const { return {}; }
    __device__ void put(unsigned n, float bd, Own, double v, double y) {
        const double qv = (double)bd * y;
        q[n] = qv;
        sum += v * qv;
    }
};

// xout = T^t u; optional clamp to [0,1] and smoothed Heaviside projection
// (Filter.cc:83-113, Filter.h:80-83)
__device__ __forceinline__ void filt_out(const FiltArgs &A, int r, const double *u) {
    const GridDesc &g = A.g;
    for (long long e = blockIdx.x * (long long)FT_N + threadIdx.x; e < g.nel(); e += (long long)gridDim.x * FT_N) {
        int i, j, k;
        lex3(e, g.ex, g.ey, i, j, k);
        double acc = 0.0;
        for (int L = 0; L < 8; L++)
            acc += u[(i + (L & 1)) + (long long)g.nx * ((j + ((L >> 1) & 1)) + (long long)g.ny * (k + (L >> 2)))];
        acc *= A.sx;
        if (A.clamp) {
            if (acc < 0.0) acc = 0.0;
            if (acc > 1.0) acc = 1.0;
        }
        A.xout[r][e] = acc;
        if (A.xphys) A.xphys[e] = project(A.proj, acc);
    }
}

// One or two filter solves: u = K^-1 (T x), then T^t u (and the projection).
// FP64 iterative refinement: the residual b - K u and u in FP64, each
// correction by Jacobi CG in FP32 on the residual scaled to unit mean square
// (GB300 runs FP64 at 1/64 of its FP32 rate).  Convergence is decided on the
// FP64 residual.  In one cooperative kernel, and CG in the form with one set
// of sums per iteration (Chronopoulos and Gear): with z = Dinv r, w = A z,
//   s = w + beta s, r = r - alpha s, p = z + beta p, d = d + alpha p,
//   gamma = r.z, delta = w.z -> beta, alpha
// where the new r of the neighbours is formed while staging, so an iteration
// is one pass and one grid barrier.  Filter and chain rule of three fields take
// 2.6 ms at 192x96x96 and 0.35 ms at 48x24x24, against 13.7 and 1.49 ms of FP64 CG
// with three launches an iteration and 64 FP64 multiply-adds a node; the result
// is 3.1e-11 instead of 4.5e-11 from the exact one at rtol 1e-10.
// What corrections cannot solve is left to k_filt_cg (filt_in_fp64, filt_judge).
__global__ void __launch_bounds__(FT_N, 3) k_filt_solve(const FiltArgs A) {
    constexpr int NV = 3;
    __shared__ __align__(16) FiltSmem sm;
    __shared__ double sred64[FT_N], stot64[FILT_RHS];
    __shared__ float sred[FILT_RHS][NV * FT_N / 32], stot[FILT_RHS * NV];
    __shared__ FiltRhs R[FILT_RHS];
    __shared__ int s_status;
    const GridDesc g = A.g;
    const long long nn = g.nn();
    const long long t0 = blockIdx.x * (long long)FT_N + threadIdx.x, ts = (long long)gridDim.x * FT_N;
    unsigned arrivals = 0;
    int slot = 0;
    // CTA sums of right-hand side r; after finish() their grid sums stand in stot[NV r + v]
    float *pf = reinterpret_cast<float *>(A.part + 2 * (size_t)FILT_RHS * gridDim.x);
    auto sums = [&](int r, const float *v) {
        cta_sums<FT_N, NV>(v, sred[r], pf + (size_t)(slot * FILT_RHS + r) * NV * gridDim.x + blockIdx.x, gridDim.x);
    };
    auto finish = [&]() {
        if (!grid_sync(A.bar, arrivals)) return false;
        grid_totals<FT_N>(pf + (size_t)slot * FILT_RHS * NV * gridDim.x, A.nr * NV, stot);
        slot ^= 1;
        return true;
    };
    // the same for one FP64 value each
    auto sum64 = [&](int r, double v) {
        cta_sums<FT_N, 1>(&v, sred64, A.part + (size_t)(slot * FILT_RHS + r) * gridDim.x + blockIdx.x, gridDim.x);
        __syncthreads();
    };
    auto finish64 = [&]() {
        if (!grid_sync(A.bar, arrivals)) return false;
        grid_totals<FT_N>(A.part + (size_t)slot * FILT_RHS * gridDim.x, A.nr, stot64);
        slot ^= 1;
        return true;
    };
    const float dinv = 1.0f / A.Kf.c[0];

    // right-hand sides b = T x, u = 0, r = b
    for (int r = 0; r < A.nr; r++) {
        double bb = 0.0;
        for (long long n = t0; n < nn; n += ts) {
            int i, j, k;
            lex3(n, g.nx, g.ny, i, j, k);
            double acc = 0.0;
            for (int c = 0; c < 8; c++) {
                const int ei = i - (c & 1), ej = j - ((c >> 1) & 1), ek = k - (c >> 2);
                if (ei < 0 || ej < 0 || ek < 0 || ei >= g.ex || ej >= g.ey || ek >= g.ez) continue;
                acc += A.xin[r][ei + (long long)g.ex * (ej + (long long)g.ey * ek)];
            }
            acc *= A.sb;
            A.b[r][n] = acc;
            A.r[r][n] = acc;
            A.u[r][0][n] = 0.0;
            bb += acc * acc;
        }
        sum64(r, bb);
    }
    if (!finish64()) return;
    if (threadIdx.x == 0) {
        s_status = TOPO_OK;
        for (int r = 0; r < FILT_RHS; r++) {
            R[r].done = 1;
            R[r].hard = 0;
            if (r >= A.nr) continue;
            R[r].bb = R[r].rr = stot64[r];
            R[r].done = stot64[r] == 0.0;
            R[r].hard = A.fp64 && !R[r].done;
            if (!isfinite(stot64[r])) s_status = TOPO_ERR_NAN;
        }
    }
    __syncthreads();
    int its = 0, ub = 0;  // ub: which u is current
    auto out = [&](int r) { return R[r].done || R[r].hard; };
    while (s_status == TOPO_OK && !(out(0) && out(1))) {
        if (threadIdx.x < FILT_RHS && !out(threadIdx.x)) R[threadIdx.x].rms = sqrt(R[threadIdx.x].rr / (double)nn);
        __syncthreads();
        // r32 = r / rms(r), z, w = K z, correction 0
        for (int r = 0; r < A.nr; r++) {
            if (out(r)) continue;
            FiltStart f{A.r[r], scale_split(1.0 / R[r].rms), dinv, A.r32[r][0], A.w32[r][0], A.d32[r], {}};
            filt_apply<float>(A, A.Kf, sm, f);
            sums(r, f.sum);
        }
        if (!finish()) return;
        if (threadIdx.x < FILT_RHS)
            filt_begin(R[threadIdx.x], stot[NV * threadIdx.x], stot[NV * threadIdx.x + 1], A.tol, nn);
        __syncthreads();
        // to the goal: a limit of its own would restart CG on the way (128 h at 48x24x24
        // 704 instead of 372 iterations with 64)
        for (int it = 0; !(R[0].idle && R[1].idle) && its < A.maxit; it++, its++) {
            const int o = it & 1, w = o ^ 1;  // buffers read and written
            for (int r = 0; r < A.nr; r++) {
                if (R[r].idle) continue;
                FiltIter f{R[r].alpha, R[r].beta, dinv, A.r32[r][o], A.s32[r][o], A.w32[r][o],
                           A.r32[r][w], A.s32[r][w], A.w32[r][w], A.p32[r], A.d32[r], {}};
                filt_apply<float>(A, A.Kf, sm, f);
                sums(r, f.sum);
            }
            if (!finish()) return;
            if (threadIdx.x < A.nr) filt_advance(R[threadIdx.x], stot + NV * threadIdx.x);
            __syncthreads();
        }
        // u += d / sigma (into the other buffer), r = b - K u, r.r
        for (int r = 0; r < A.nr; r++) {
            if (R[r].done) {  // converged earlier: carried along
                for (long long n = t0; n < nn; n += ts) A.u[r][ub ^ 1][n] = A.u[r][ub][n];
                continue;
            }
            if (R[r].hard) continue;
            FiltResid f{A.u[r][ub], A.b[r], A.d32[r], R[r].rms, A.u[r][ub ^ 1], A.r[r], 0.0};
            filt_apply<double>(A, A.Kd, sm, f);
            sum64(r, f.sum);
        }
        if (!finish64()) return;
        ub ^= 1;
        if (threadIdx.x < A.nr) filt_judge(R[threadIdx.x], stot64[threadIdx.x], A.tol, its, A.maxit);
        __syncthreads();
    }
    const int status = s_status;
    if (status == TOPO_OK && !R[0].hard && !R[1].hard) {
        for (int r = 0; r < A.nr; r++) filt_out(A, r, A.u[r][ub]);
    }
    if (grid_leave(A.bar)) {
        A.out->status = status;
        A.out->hard = (R[0].hard ? 1 : 0) | (R[1].hard ? 2 : 0);
        A.out->cur = ub;
        __threadfence_system();
    }
}

// Jacobi CG in FP64 on right-hand side r, whose b = T x stands in A.b[r], from u = 0:
// the product, the update and the direction in turn, a grid barrier after each.  A
// kernel of its own: within k_filt_solve it cost that one 5% in registers.
__global__ void __launch_bounds__(FT_N, 3) k_filt_cg(const FiltArgs A, int r) {
    __shared__ __align__(16) FiltSmem sm;
    __shared__ double sred[FT_N], stot[2], bb;
    __shared__ FiltCg cg;
    const GridDesc g = A.g;
    const long long nn = g.nn(), t0 = blockIdx.x * (long long)FT_N + threadIdx.x, ts = (long long)gridDim.x * FT_N;
    unsigned arrivals = 0;
    int slot = 0;
    auto reduce = [&](double v0, double v1) {  // grid sums into stot
        double *part = A.part + (size_t)slot * 2 * gridDim.x;
        cta_sums<FT_N, 1>(&v0, sred, part + blockIdx.x, gridDim.x);
        __syncthreads();
        cta_sums<FT_N, 1>(&v1, sred, part + gridDim.x + blockIdx.x, gridDim.x);
        if (!grid_sync(A.bar, arrivals)) return false;
        grid_totals<FT_N>(part, 2, stot);
        slot ^= 1;
        return true;
    };
    const double dinv = 1.0 / A.Kd.c[0];
    auto prec = [&](long long n, double v) {  // Dinv v
        int i, j, k;
        lex3(n, g.nx, g.ny, i, j, k);
        const int ends = (i == 0 || i == g.nx - 1) + (j == 0 || j == g.ny - 1) + (k == 0 || k == g.nz - 1);
        return v * (dinv * (double)(1 << ends));
    };
    double *x = A.u[r][0], *p = A.u[r][1], *res = A.r[r], *q = A.q[r];
    double s0 = 0.0, s1 = 0.0;
    for (long long n = t0; n < nn; n += ts) {
        const double b = A.b[r][n], z = prec(n, b);
        x[n] = 0.0;
        res[n] = b;
        p[n] = z;
        s0 += b * b;
        s1 += b * z;
    }
    if (!reduce(s0, s1)) return;
    if (threadIdx.x == 0) {
        bb = stot[0];
        filt_cg_begin(cg, stot[1]);
    }
    __syncthreads();
    for (;;) {
        FiltMul f{p, q, 0.0};
        filt_apply<double>(A, A.Kd, sm, f);
        if (!reduce(f.sum, 0.0)) return;
        if (threadIdx.x == 0) filt_cg_step(cg, stot[0]);
        __syncthreads();
        if (cg.done) break;
        const double al = cg.alpha;
        s0 = s1 = 0.0;
        for (long long n = t0; n < nn; n += ts) {
            x[n] += al * p[n];
            const double v = res[n] - al * q[n];
            res[n] = v;
            s0 += v * v;
            s1 += v * prec(n, v);
        }
        if (!reduce(s0, s1)) return;
        if (threadIdx.x == 0) filt_cg_judge(cg, stot[0], stot[1], A.tol, bb, A.maxit);
        __syncthreads();
        if (cg.done) break;
        const double be = cg.beta;
        for (long long n = t0; n < nn; n += ts) p[n] = prec(n, res[n]) + be * p[n];
        if (!grid_sync(A.bar, arrivals)) return;
    }
    if (grid_leave(A.bar)) {
        A.out->status = cg.status;
        __threadfence_system();
    }
}

static __global__ void k_filt_out(const FiltArgs A, int r, const double *u) { filt_out(A, r, u); }

struct TopoPDEFilt {
    GridDesc g;
    int nrhs;        // right-hand sides that the workspace is for
    FiltArgs args;   // operator, buffers and layout of the launches
    unsigned grid;   // CTAs of k_filt_solve: as many as are resident at once, at most one per run
    double *mnd;
    double *part;
    unsigned int *counter;  // [0] reductions, [1..3] the grid barrier
    FiltStatus *status;     // mapped host memory
    std::vector<void *> ptrs;
    cudaStream_t stream;
};

// Filter::Gradients chain rule of the projection (Filter.cc:128-169)
__global__ void k_chain(long long nel, const double *__restrict__ xt, double *df, int m, double *dg, Projection pr) {
    for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < nel; e += (long long)gridDim.x * blockDim.x) {
        const double d = project_slope(pr, xt[e]);
        df[e] *= d;
        for (int j = 0; j < m; j++) dg[(long long)j * nel + e] *= d;
    }
}

// GetMND (Filter.cc:208-227)
__global__ void k_mnd(long long n, const double *__restrict__ x, Partials<1> part, double *out) {
    double v[1] = {0.0};
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        v[0] += 4.0 * x[i] * (1.0 - x[i]);
    double tot[1];
    if (grid_reduce<EW, 1>(v, part, tot)) *out = tot[0] / (double)n;
}

// ---------------------------------------------------------------------------
int pdefilt_create(TopoPDEFilt **out, int nx, int ny, int nz, double hx, double hy, double hz, double rmin, double rtol,
                   int maxit, int nrhs) {
    *out = nullptr;
    if (nx < 2 || ny < 2 || nz < 2 || hx <= 0 || hy <= 0 || hz <= 0 || rmin <= 0) {
        set_error("invalid PDE filter parameters");
        return TOPO_ERR_ARG;
    }
    TopoPDEFilt *f = new TopoPDEFilt();
    f->g = GridDesc{nx, ny, nz, nx - 1, ny - 1, nz - 1};
    const double R = rmin / 2.0 / sqrt(3.0);  // PDEFilter.cc:32
    f->nrhs = nrhs;
    const double hh[3] = {hx, hy, hz};
    filt_stencil(hh, R, f->args.Kd.c);
    for (int S = 0; S < 8; S++) f->args.Kf.c[S] = (float)f->args.Kd.c[S];
    cudaError_t e = cudaStreamCreateWithFlags(&f->stream, cudaStreamNonBlocking);
    if (e != cudaSuccess) {
        set_error(std::string("cudaStreamCreate: ") + cudaGetErrorString(e));
        delete f;
        return TOPO_ERR_CUDA;
    }
    const long long nn = f->g.nn();
    // one allocation for the workspace: 27 of their own made the set-up at
    // 192x96x96 1.9 instead of under 1.2 ms
    FiltArgs &A = f->args;
    A.g = f->g;
    std::vector<std::pair<void **, size_t>> want;
    auto get = [&](auto **p, size_t n) { want.emplace_back((void **)p, sizeof(**p) * n); };
    for (int r = 0; r < nrhs; r++) {
        for (int k = 0; k < 2; k++) {
            get(&A.u[r][k], nn);
            for (float **q : {&A.s32[r][k], &A.w32[r][k]}) get(q, nn);
        }
        for (double **q : {&A.b[r], &A.r[r], &A.q[r]}) get(q, nn);
        for (float **q : {&A.p32[r], &A.d32[r]}) get(q, nn);
    }
    get(&f->mnd, 1);
    get(&f->part, 2 * 65536);
    get(&f->counter, 4);
    size_t bytes = 0;
    for (const auto &w : want) bytes += (w.second + 255) / 256 * 256;
    char *mem = nullptr;
    int rc = cudaMalloc((void **)&mem, bytes) != cudaSuccess;
    if (rc) {
        cudaGetLastError();
        set_error("cudaMalloc failed in PDE filter");
    } else {
        f->ptrs.push_back(mem);
        cudaMemset(mem, 0, bytes);
        for (const auto &w : want) {
            *w.first = mem;
            mem += (w.second + 255) / 256 * 256;
        }
        for (int r = 0; r < nrhs; r++) {
            A.r32[r][0] = (float *)A.q[r];
            A.r32[r][1] = A.r32[r][0] + nn;
        }
    }
    if (rc) {
        pdefilt_destroy(f);
        return TOPO_ERR_OOM;
    }
    e = cudaHostAlloc((void **)&f->status, sizeof(FiltStatus), cudaHostAllocMapped);
    if (e == cudaSuccess) e = cudaHostGetDevicePointer((void **)&A.out, f->status, 0);
    // resident CTAs, and runs of planes that give each about one: a run reads two planes more than it completes
    int dev = 0, nsm = 0, per_sm = 0, per_cg = 0;
    if (e == cudaSuccess) e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_filt_solve, FT_N, 0);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_cg, k_filt_cg, FT_N, 0);
    if (e == cudaSuccess) e = cudaStreamSynchronize(f->stream);
    if (e != cudaSuccess || per_sm < 1 || per_cg < 1) {
        set_error(std::string("PDE filter setup: ") + cudaGetErrorString(e));
        pdefilt_destroy(f);
        return TOPO_ERR_CUDA;
    }
    const int resident = std::min(per_sm, per_cg) * nsm;
    const Patch pt = plane_patch(nx, ny, FT_N, 1, FT_PLANE);
    A.tx = pt.tx;
    A.ty = pt.ty;
    A.ntx = pt.ntx;
    A.nty = pt.nty;
    const int runs = std::max(1, std::min(nz, resident / std::max(1, A.ntx * A.nty)));
    A.cz = (nz + runs - 1) / runs;
    A.ncz = (nz + A.cz - 1) / A.cz;
    f->grid = (unsigned)std::min(resident, A.ntx * A.nty * A.ncz);
    const int ve = std::max(-1000, std::min(1000, std::ilogb(hx * hy * hz)));
    A.sb = std::ldexp(0.125, ve);
    A.sx = std::ldexp(0.125, -ve);
    A.tol = rtol;
    A.maxit = maxit;
    A.fp64 = filt_in_fp64(hh, R, rtol);
    A.part = f->part;
    A.bar = GridBar{f->counter + 1, f->counter + 2, f->counter + 3};
    *out = f;
    return TOPO_OK;
}

void pdefilt_destroy(TopoPDEFilt *f) {
    if (!f) return;
    for (void *p : f->ptrs) cudaFree(p);
    if (f->status) cudaFreeHost(f->status);
    if (f->stream) cudaStreamDestroy(f->stream);
    delete f;
}

long long pdefilt_nel(const TopoPDEFilt *f) { return f->g.nel(); }

// results of up to FILT_RHS element fields, in place allowed (every input is
// read before the first result is written)
static int filt_solve(TopoPDEFilt *f, int nr, const double *const *xin, double *const *xout, double *xphys, int clamp,
                      int projection, double beta, double eta) {
    cudaStream_t s = f->stream;
    FiltArgs A = f->args;
    A.nr = nr;
    for (int r = 0; r < nr; r++) {
        A.xin[r] = xin[r];
        A.xout[r] = xout[r];
    }
    A.xphys = xphys;
    A.clamp = clamp;
    A.proj = make_projection(projection, beta, eta);
    auto launch = [&](const void *kernel, void **args) {
        f->status->status = TOPO_ERR_CUDA;
        count_launch();
        const cudaError_t e = cudaLaunchCooperativeKernel(kernel, dim3(f->grid), dim3(FT_N), args, 0, s);
        return e == cudaSuccess ? cudaStreamSynchronize(s) : e;
    };
    void *args[] = {&A};
    FCK(launch((const void *)k_filt_solve, args));
    int st = *(volatile int *)&f->status->status;
    const int hard = f->status->hard, cur = f->status->cur;
    if (st == TOPO_OK && hard) {
        for (int r = 0; r < nr && st == TOPO_OK; r++) {
            if (!((hard >> r) & 1)) continue;
            void *cargs[] = {&A, &r};
            FCK(launch((const void *)k_filt_cg, cargs));
            st = *(volatile int *)&f->status->status;
        }
        for (int r = 0; r < nr && st == TOPO_OK; r++) {  // no result before all are solved
            count_launch();
            k_filt_out<<<f->grid, FT_N, 0, s>>>(A, r, A.u[r][(hard >> r) & 1 ? 0 : cur]);
        }
        FCK(cudaGetLastError());
        FCK(cudaStreamSynchronize(s));
    }
    if (st == TOPO_OK) return TOPO_OK;
    if (st == TOPO_ERR_CUDA) {  // the grid barrier gave up
        FCK(cudaMemsetAsync(f->counter + 1, 0, 3 * sizeof(unsigned), s));
        FCK(cudaStreamSynchronize(s));
        set_error("PDE filter: the solve's grid barrier ran out of time");
    } else {
        set_error(std::string("PDE filter solve failed with status ") + std::to_string(st));
    }
    return st;
}

int pdefilt_apply_dev(TopoPDEFilt *f, const double *x_dev, double *xout_dev) {
    return filt_solve(f, 1, &x_dev, &xout_dev, nullptr, 0, 0, 0.0, 0.0);
}

int filter_project_dev(TopoPDEFilt *f, const double *x_dev, double *xTilde_dev, double *xPhys_dev, int projection,
                       double beta, double eta) {
    return filt_solve(f, 1, &x_dev, &xTilde_dev, xPhys_dev, 1, projection, beta, eta);
}

int filter_gradients_dev(TopoPDEFilt *f, const double *xTilde_dev, double *dfdx_dev, int m, double *dgdx_dev,
                         int projection, double beta, double eta) {
    long long nel = f->g.nel();
    if (projection) {
        count_launch();
        k_chain<<<ew_blocks(nel), EW, 0, f->stream>>>(nel, xTilde_dev, dfdx_dev, m, dgdx_dev,
                                                         make_projection(1, beta, eta));
    }
    // PDEFilt::Gradients == FilterProject (PDEFilter.cc:224), dfdx and the m columns of dgdx
    for (int j = 0; j <= m; j += f->nrhs) {
        double *v[FILT_RHS];
        int nr = 0;
        for (; nr < f->nrhs && j + nr <= m; nr++) v[nr] = j + nr == 0 ? dfdx_dev : dgdx_dev + (size_t)(j + nr - 1) * nel;
        const int rc = filt_solve(f, nr, v, v, nullptr, 0, 0, 0.0, 0.0);
        if (rc) return rc;
    }
    return TOPO_OK;
}

int filter_mnd_dev(TopoPDEFilt *f, const double *x_dev, double *mnd) {
    long long nel = f->g.nel();
    Partials<1> p1{f->part, f->counter};
    count_launch();
    k_mnd<<<red_blocks(nel), EW, 0, f->stream>>>(nel, x_dev, p1, f->mnd);
    FCK(cudaMemcpyAsync(mnd, f->mnd, sizeof(double), cudaMemcpyDeviceToHost, f->stream));
    FCK(cudaStreamSynchronize(f->stream));
    return TOPO_OK;
}

}  // namespace topo
