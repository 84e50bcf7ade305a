// march.cuh -- the matrix-free hex8 operator in FP64: columns of elements
// marched along z.
//
// A CTA owns a TX x TY patch of element columns, one column per thread, and a
// run of node layers.  Per element layer a thread
//   1. reads the 4 corner nodes of its column on the upper node layer from
//      shared memory and forms their 12 in-plane modes (sums and differences
//      along x, then y); those of the lower layer are the previous step's, kept
//      in registers;
//   2. combines the two layers along z, applies the element operator in the
//      mode basis (common.cuh) and transforms back along z: the lower half is
//      added to the upper half that the element below left in registers, which
//      completes the in-plane modes of this column's share of the lower layer;
//   3. transforms back along y and hands the far half to the column at y + 1
//      through shared memory; transforms back along x and hands the far half
//      to the column at x + 1 by a warp shuffle.
// Step 3 leaves the assembled value of node (ex, ey) of the lower layer in the
// thread of column (ex, ey): no element output is stored anywhere, and there
// are no atomics, so results are bitwise reproducible.
//
// Why: the FP64 products are bound by FP64 instructions (GB300: 2 lanes a clock
// and SM, measured), not by memory.  Sharing the in-plane stages between the
// elements above and below a node layer and completing the sums of neighbours
// before the next stage takes 111 sums an element where transforming every
// element on its own takes 165, the element math of equal-edged boxes 57
// instructions instead of 98, and the columns on the patch's rim with one
// element layer a run are the only work done twice, against 1.49 times all of it
// for bricks of 7^3 output nodes.
//
// The node layer two steps ahead is loaded into registers while the current
// layer is computed and stored to the free one of two shared-memory layers,
// so one barrier per layer orders everything.
#pragma once
#include "common.cuh"

namespace topo {

// Policy interface (tile.cuh's policies, T = double), besides HAS_K, HAS_M,
// NRED, w, pre, epilogue, finish and part:
//   static constexpr int M_SRC, M_IN;     staged arrays; vectors formed of them: with
//                                         M_IN = 2, K acts on the first and M on the second
//   const double *msrc(int a) const;      staged array a, 3 values per node
//   void mval(const double raw[M_SRC], double v[M_IN]) const;
//   const uint8_t *mmask() const;         clamp bits of the staged values, or null

constexpr int MARCH_THREADS = 192;  // largest patch
constexpr int MARCH_SLOTS = 5;      // staged nodes' values per thread and layer (march_config keeps to it)

struct MarchDims {
    int tx, ty;    // patch: element columns along x (8, 16 or 32) and y
    int ntx, nty;  // patches: each completes (tx - 1) x (ty - 1) nodes of a layer
    int cz, ncz;   // node layers per run, runs
};
__host__ __device__ constexpr size_t march_smem_bytes(int tx, int ty, int nin) {
    return sizeof(double) * (2 * (size_t)nin * (tx + 1) * (ty + 1) * 3 + 2 * (size_t)6 * tx * ty);
}

// in-plane modes F[c][m], m = (x difference) + 2 (y difference), of the four
// nodes at s, s + 1, s + row, s + row + 1 of a staged layer
__device__ __forceinline__ void march_face(const double *lay, int s, int row, double F[3][4]) {
#pragma unroll
    for (int c = 0; c < 3; c++) {
        const double a0 = lay[3 * s + c], a1 = lay[3 * (s + 1) + c];
        const double b0 = lay[3 * (s + row) + c], b1 = lay[3 * (s + row + 1) + c];
        const double sa = a0 + a1, da = a1 - a0, sb = b0 + b1, db = b1 - b0;
        F[c][0] = sa + sb;
        F[c][1] = da + db;
        F[c][2] = sb - sa;
        F[c][3] = db - da;
    }
}

// CUBE: elements with three equal edges
template <class Pol, bool CUBE>
__global__ void __launch_bounds__(MARCH_THREADS, Pol::M_IN == 1 ? 2 : 1)
    k_march(const GridDesc g, const ElemConst<double> C, const Pol pol, const MarchDims D) {
    grid_dep_wait();
    TOPO_DYNAMIC_SMEM(double, lay0);
    constexpr int NIN = Pol::M_IN, NSRC = Pol::M_SRC;
    const int tid = threadIdx.x, NT = D.tx * D.ty;
    const int ly = tid / D.tx, lx = tid - ly * D.tx;
    const int row = D.tx + 1, nst = 3 * row * (D.ty + 1);  // staged values per layer and vector
    double *xch = lay0 + 2 * NIN * nst;                    // two buffers of 6 values per thread
    int b = blockIdx.x;
    const int bx = b % D.ntx;
    b /= D.ntx;
    const int by = b % D.nty, bz = b / D.nty;
    const int ex = bx * (D.tx - 1) - 1 + lx, ey = by * (D.ty - 1) - 1 + ly;
    const int k0 = bz * D.cz, k1 = min(k0 + D.cz, g.nz);
    const long long plane = (long long)g.nx * g.ny;
    // staged values of this thread: index within a node plane, or -1 outside
    int slot[MARCH_SLOTS];
#pragma unroll
    for (int q = 0; q < MARCH_SLOTS; q++) {
        const int v = tid + q * NT, r = v / (3 * row), w = v - r * 3 * row;
        const int gx = bx * (D.tx - 1) - 1 + w / 3, gy = by * (D.ty - 1) - 1 + r;
        slot[q] = (v < nst && gx >= 0 && gx < g.nx && gy >= 0 && gy < g.ny) ? 3 * (gx + g.nx * gy) + w % 3 : -1;
    }
    const uint8_t *mask = pol.mmask();
    // a node layer into registers (r, and the clamp bits f), and from there to shared memory
    auto fetch = [&](int k, double r[MARCH_SLOTS][NSRC], uint8_t f[MARCH_SLOTS]) {
        const bool in = k >= 0 && k < g.nz;
#pragma unroll
        for (int q = 0; q < MARCH_SLOTS; q++) {
            const bool ok = in && slot[q] >= 0;
#pragma unroll
            for (int a = 0; a < NSRC; a++) r[q][a] = ok ? pol.msrc(a)[3 * plane * k + slot[q]] : 0.0;
            f[q] = ok && mask ? mask[plane * k + slot[q] / 3] : 0;
        }
    };
    auto store = [&](int k, const double r[MARCH_SLOTS][NSRC], const uint8_t f[MARCH_SLOTS]) {
        double *lay = lay0 + (k & 1) * NIN * nst;
#pragma unroll
        for (int q = 0; q < MARCH_SLOTS; q++) {
            const int v = tid + q * NT;
            if (v >= nst) continue;
            double t[NIN];
            pol.mval(r[q], t);
            const bool fx = (f[q] >> ((unsigned)slot[q] % 3u)) & 1;  // a clamped value is staged as zero (f is 0 outside)
#pragma unroll
            for (int n = 0; n < NIN; n++) lay[n * nst + v] = fx ? 0.0 : t[n];
        }
    };
    const bool col = ex >= 0 && ex < g.ex && ey >= 0 && ey < g.ey;
    const long long ecol = ex + (long long)g.ex * ey, eplane = (long long)g.ex * g.ey;
    auto weights = [&](int k, double &ck, double &cm) {  // element layer k
        ck = 0.0;
        cm = 0.0;
        if (col && k >= 0 && k < g.ez) pol.w.get(ecol + eplane * k, ck, cm);
    };
    const bool out = lx > 0 && ly > 0 && ex < g.nx && ey < g.ny;
    const bool any = __any_sync(0xffffffffu, col);  // else the warp's columns are all outside
    double red[Pol::NRED > 0 ? Pol::NRED : 1];
#pragma unroll
    for (int r = 0; r < (Pol::NRED > 0 ? Pol::NRED : 1); r++) red[r] = 0.0;

    double raw[MARCH_SLOTS][NSRC], ck, cm;
    uint8_t fix[MARCH_SLOTS];
    {
        double raw0[MARCH_SLOTS][NSRC];
        uint8_t fix0[MARCH_SLOTS];
        fetch(k0 - 1, raw0, fix0);
        fetch(k0, raw, fix);
        weights(k0 - 1, ck, cm);
        store(k0 - 1, raw0, fix0);
        store(k0, raw, fix);
    }
    __syncthreads();
    const int sn = lx + row * ly;
    double F[NIN][3][4], carry[3][4];
#pragma unroll
    for (int n = 0; n < NIN; n++) march_face(lay0 + (((k0 - 1) & 1) * NIN + n) * nst, sn, row, F[n]);
#pragma unroll
    for (int c = 0; c < 3; c++)
#pragma unroll
        for (int m = 0; m < 4; m++) carry[c][m] = 0.0;
    __syncthreads();  // layer k0 - 1 is free

    for (int k = k0 - 1; k < k1; k++) {  // element layer k, between node layers k and k + 1
        if (k + 2 <= k1) fetch(k + 2, raw, fix);
        double ckn, cmn;
        weights(k + 1, ckn, cmn);
        const long long n = ex + (long long)g.nx * ey + plane * k;
        const bool emit = out && k >= k0;
        const auto pre = pol_pre(pol, emit ? n : 0, 0);
        double G[3][4];  // lower modes: this column's completed share of node layer k
        {
            double N[NIN][3][4];
#pragma unroll
            for (int i = 0; i < NIN; i++) march_face(lay0 + (((k + 1) & 1) * NIN + i) * nst, sn, row, N[i]);
            if (any && k >= 0 && k < g.ez) {
                double U[3][8], Y[3][8];
#pragma unroll
                for (int c = 0; c < 3; c++)
#pragma unroll
                    for (int m = 0; m < 4; m++) {
                        U[c][m] = F[0][c][m] + N[0][c][m];
                        U[c][m | 4] = N[0][c][m] - F[0][c][m];
                    }
                mode_apply<CUBE, Pol::HAS_K, Pol::HAS_M && NIN == 1>(C, ck, cm, U, Y);
                if constexpr (NIN == 2) {
#pragma unroll
                    for (int m = 0; m < 4; m++) {
                        const double ws = cm * C.W[m], wd = cm * C.W[m | 4];
#pragma unroll
                        for (int c = 0; c < 3; c++) {
                            Y[c][m] += ws * (F[1][c][m] + N[1][c][m]);
                            Y[c][m | 4] += wd * (N[1][c][m] - F[1][c][m]);
                        }
                    }
                }
#pragma unroll
                for (int c = 0; c < 3; c++)
#pragma unroll
                    for (int m = 0; m < 4; m++) {
                        G[c][m] = carry[c][m] + (Y[c][m] - Y[c][m | 4]);
                        carry[c][m] = Y[c][m] + Y[c][m | 4];
                    }
            } else {
#pragma unroll
                for (int c = 0; c < 3; c++)
#pragma unroll
                    for (int m = 0; m < 4; m++) {
                        G[c][m] = carry[c][m];
                        carry[c][m] = 0.0;
                    }
            }
#pragma unroll
            for (int i = 0; i < NIN; i++)
#pragma unroll
                for (int c = 0; c < 3; c++)
#pragma unroll
                    for (int m = 0; m < 4; m++) F[i][c][m] = N[i][c][m];
        }
        // back along y: the near half stays (G[c][0..1]), the far half goes to the column at y + 1
        double *xb = xch + (k & 1) * 6 * NT;
#pragma unroll
        for (int c = 0; c < 3; c++)
#pragma unroll
            for (int m = 0; m < 2; m++) {
                xb[(2 * c + m) * NT + tid] = G[c][m] + G[c][m | 2];
                G[c][m] = G[c][m] - G[c][m | 2];
            }
        if (k + 2 <= k1) store(k + 2, raw, fix);
        ck = ckn;
        cm = cmn;
        __syncthreads();
        double y[3];
#pragma unroll
        for (int c = 0; c < 3; c++) {
            if (ly > 0) {
                G[c][0] += xb[(2 * c) * NT + tid - D.tx];
                G[c][1] += xb[(2 * c + 1) * NT + tid - D.tx];
            }
            // back along x: the far half goes to the column at x + 1
            y[c] = (G[c][0] - G[c][1]) + __shfl_up_sync(0xffffffffu, G[c][0] + G[c][1], 1, D.tx);
        }
        if (emit) pol_epi(pol, n, ex, ey, k, y, red, pre, 0);
    }
    if constexpr (Pol::NRED > 0) {
        double tot[Pol::NRED];
        if (grid_reduce64<MARCH_THREADS, Pol::NRED>(red, pol.part, tot, NT)) pol.finish(tot);
    }
}

// Patch and run lengths of a grid.  Each of an SM's four schedulers issues an
// FP64 instruction of a warp every 64 clocks, so the unit here is an element
// layer of up to four warps, about 170 x 64 clocks, whole when fewer are there;
// a layer's barrier and load latency add about 0.15 units to every wave of
// resident CTAs (12 warps of 168 registers an SM), a CTA's start 0.3.  So a wide
// grid takes patches with little rim and long runs, a small one spreads over the
// SMs in patches of four warps with runs as short as one layer.
inline MarchDims march_config(const GridDesc &g, int nsm) {
    MarchDims best{};
    double best_t = 1e300;
    for (int tx = 32; tx >= 8; tx /= 2)
        for (int ty = MARCH_THREADS / tx; ty >= 2; ty--) {
            if ((tx * ty) % 32 || 3 * (tx + 1) * (ty + 1) > MARCH_SLOTS * tx * ty) continue;
            MarchDims d;
            d.tx = tx;
            d.ty = ty;
            d.ntx = (g.nx + tx - 2) / (tx - 1);
            d.nty = (g.ny + ty - 2) / (ty - 1);
            const int warps = tx * ty / 32, fit = 12 / warps;
            for (int runs = 1; runs <= g.nz; runs++) {
                d.cz = (g.nz + runs - 1) / runs;
                d.ncz = (g.nz + d.cz - 1) / d.cz;
                if (d.ncz < runs) continue;
                const long long ctas = (long long)d.ntx * d.nty * d.ncz, per_sm = (ctas + nsm - 1) / nsm;
                const double layers = d.cz + 1;
                const double t = (double)((per_sm * warps + 3) / 4) * layers +
                                 (double)((per_sm + fit - 1) / fit) * (0.15 * layers + 0.3);
                if (t < best_t * (1 - 1e-9)) {
                    best_t = t;
                    best = d;
                }
            }
        }
    return best;
}

}  // namespace topo
