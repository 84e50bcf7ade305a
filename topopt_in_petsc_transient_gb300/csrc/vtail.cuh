// vtail.cuh -- the last smoothed level of the FP32 V-cycle and the dense coarse
// solve below it in one kernel.
//
// A level of at most VT_CTAS bricks gives a kernel too little work to pay for its
// launch: smoothing, residual, restriction, coarse solve and prolongation of
// 17x9x9 nodes were ten dependent launches of 2 to 6 us each.  Here one
// thread-block cluster takes all of them, a brick per CTA, with a cluster barrier
// (which orders global memory between its CTAs) between the steps.  A thread
// keeps its element's weights and its node's values in registers; only the
// staged x goes through memory.  24 us a V-cycle at 17x9x9 nodes over 9x5x5
// instead of about 50, bound by the latency of a step: staging, element and
// gather phase, barrier.  The arithmetic is that of the separate kernels
// (PolCheb, PolResid, k_cheb0), so results agree to the bit.
#pragma once
#include <cooperative_groups.h>

#include "kernels.cuh"

namespace topo {

constexpr int VT_CTAS = 16;   // largest (non-portable) cluster
constexpr int VT_SMOOTH = 16;  // most smoothing steps

struct VTail {
    GridDesc g, gc;  // the level and the coarse one
    const uint8_t *fixed, *fixc;
    Weights<float> w;
    const float *b, *dinv, *Ainv;
    float *xa, *xb, *r, *bc, *xc;  // the result is left in xb
    const float *ctab;
    int nu, n;  // smoothing steps, coarse DOFs
};
struct VTElem {  // weights of the thread's element, loaded once
    static constexpr bool HAS_K = true, HAS_M = true;
    float k, m;
    __device__ void coef(long long, float &ck, float &cm) const {
        ck = k;
        cm = m;
    }
};

static __global__ void __launch_bounds__(TILE_THREADS, 1) k_vtail(const VTail V, const ElemConst<float> C) {
    TOPO_DYNAMIC_SMEM(unsigned char, smem_raw);
    __shared__ float c12[2 * VT_SMOOTH];
    grid_dep_wait();
    const auto cl = cooperative_groups::this_cluster();
    const GridDesc &g = V.g;
    const int tid = threadIdx.x, q0 = blockIdx.x * TILE_THREADS + tid, nq = gridDim.x * TILE_THREADS;
    float *sIn = reinterpret_cast<float *>(smem_raw), *sEl = sIn + TILE_STAGED * 3;
    int ntx, nty;
    const int ntiles = tile_count(g, ntx, nty), tile = blockIdx.x;
    const bool work = tile < ntiles;
    const int i0 = (tile % ntx) * TILE, j0 = ((tile / ntx) % nty) * TILE, k0 = (tile / (ntx * nty)) * TILE;
    if (tid < 2 * V.nu) c12[tid] = V.ctab[tid];
    __syncthreads();
    // staged nodes, element and output node of this thread (tile.cuh)
    int sn[2];
    uint8_t sf[2] = {0, 0};
#pragma unroll
    for (int it = 0; it < 2; it++) {
        const int s = tid + it * TILE_THREADS;
        const int i = i0 - 1 + s % TILE_N, j = j0 - 1 + (s / TILE_N) % TILE_N, k = k0 - 1 + s / (TILE_N * TILE_N);
        const bool in = work && s < TILE_STAGED && i >= 0 && i < g.nx && j >= 0 && j < g.ny && k >= 0 && k < g.nz;
        sn[it] = in ? i + g.nx * (j + g.ny * k) : -1;
        if (in) sf[it] = V.fixed[sn[it]];
    }
    VTElem el{0.0f, 0.0f};
    {
        const int i = i0 - 1 + (tid & 7), j = j0 - 1 + ((tid >> 3) & 7), k = k0 - 1 + (tid >> 6);
        if (work && i >= 0 && i < g.ex && j >= 0 && j < g.ey && k >= 0 && k < g.ez)
            V.w.get(i + (long long)g.ex * (j + (long long)g.ey * k), el.k, el.m);
    }
    const int tx = tid % TILE, ty = (tid / TILE) % TILE, tz = tid / (TILE * TILE);
    const int oi = i0 + tx, oj = j0 + ty, ok = k0 + tz;
    const bool out = work && tid < TILE_OUT && oi < g.nx && oj < g.ny && ok < g.nz;
    const int on = out ? oi + g.nx * (oj + g.ny * ok) : 0;
    float b[3] = {0}, di[3] = {0}, d[3] = {0}, x[3] = {0};
    uint8_t f = 0;
    if (out) {
        f = V.fixed[on];
#pragma unroll
        for (int c = 0; c < 3; c++) {
            b[c] = V.b[3 * on + c];
            di[c] = V.dinv[3 * on + c];
            x[c] = d[c] = c12[1] * di[c] * b[c];  // first step from zero
        }
    }
    float *xs = V.xb, *xo = V.xa;  // last written, next
    auto put = [&] {               // the node's x for the other CTAs
        if (out)
#pragma unroll
            for (int c = 0; c < 3; c++) xo[3 * on + c] = x[c];
        float *t = xs;
        xs = xo;
        xo = t;
    };
    for (int a = 0; a < 2 * V.nu; a++) {  // nu - 1 steps, the residual, nu steps
        if (work) {
#pragma unroll
            for (int it = 0; it < 2; it++) {
                const int s = tid + it * TILE_THREADS, n = sn[it];
                float v[3] = {0.0f, 0.0f, 0.0f};
                if (n >= 0) {
#pragma unroll
                    for (int c = 0; c < 3; c++)
                        v[c] = a == 0 ? c12[1] * V.dinv[3 * n + c] * V.b[3 * n + c] : xs[3 * n + c];
                    mask3(sf[it], v);
                }
                if (s < TILE_STAGED)
#pragma unroll
                    for (int c = 0; c < 3; c++) sIn[s * 3 + c] = v[c];
            }
            __syncthreads();
            tile_elements<float>(g, C, el, sIn, sEl, i0, j0, k0);
            __syncthreads();
        }
        float y[3] = {0.0f, 0.0f, 0.0f};
        if (out) {
#pragma unroll
            for (int L = 0; L < 8; L++) {
                const int le = (tx + 1 - (L & 1)) + TILE_E * ((ty + 1 - ((L >> 1) & 1)) + TILE_E * (tz + 1 - (L >> 2)));
#pragma unroll
                for (int c = 0; c < 3; c++) y[c] = tadd(y[c], sEl[le * EL_STRIDE + L * 3 + c]);
            }
#pragma unroll
            for (int c = 0; c < 3; c++) y[c] = b[c] - (((f >> c) & 1) ? x[c] : y[c]);  // the residual
        }
        if (a != V.nu - 1) {
            const int k = a < V.nu - 1 ? a + 1 : a - V.nu;
            const float c1 = c12[2 * k], c2 = c12[2 * k + 1];
#pragma unroll
            for (int c = 0; c < 3; c++) {
                if (k == 0) d[c] = 0.0f;
                d[c] = c1 * d[c] + c2 * di[c] * y[c];
                x[c] = x[c] + d[c];
            }
        } else {
            if (out)
#pragma unroll
                for (int c = 0; c < 3; c++) V.r[3 * on + c] = y[c];
            cl.sync();
            restrict_range(g, V.gc, V.fixc, V.r, V.bc, q0, nq);
            cl.sync();
            gemv_range<3>(V.n, V.Ainv, V.bc, V.xc, q0 >> 5, nq >> 5);
            cl.sync();
            if (out) prolong_node(V.gc, V.xc, oi, oj, ok, f, x);
        }
        put();
        cl.sync();
    }
}

}  // namespace topo
