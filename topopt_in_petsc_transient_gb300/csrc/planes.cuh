// planes.cuh -- what the filters share: patches of a plane, and the smoothed
// Heaviside projection.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

namespace topo {

// Patch of tx x ty columns, at most nt of them, that covers an nx x ny plane
// (ntx x nty patches) with the fewest idle threads; `halo` columns around it
// are staged too, at most `most` values in all.  Node counts are one more than
// round numbers, where a fixed 32 x 8 patch idles a seventh of a plane of 193.
struct Patch {
    int tx, ty, ntx, nty;
};
inline Patch plane_patch(int nx, int ny, int nt, int halo, int most) {
    Patch b{1, 1, nx, ny};
    double best = 0.0;
    for (int t = 64; t >= 16; t--) {  // wide ones first: a narrower one has to be 2% better
        const int ntx = (nx + t - 1) / t, tx = (nx + ntx - 1) / ntx;
        const int cap = std::min(nt / tx, most / (tx + 2 * halo) - 2 * halo);
        if (cap < 1) continue;
        const int nty = (ny + cap - 1) / cap, ty = (ny + nty - 1) / nty;
        const double use = (double)nx * ny / ((double)ntx * nty * nt);
        if (use <= best * 1.02) continue;
        best = use;
        b = Patch{tx, ty, ntx, nty};
    }
    return b;
}

// Smoothed Heaviside projection (Filter.h:80-88) with one exponential and one
// quotient: E = exp(-2 |v|), tanh v = +-(1 - E) / (1 + E), 1 - tanh^2 v =
// 4 E / (1 + E)^2.  FP64 runs at 2 lanes a clock and SM here, and tanh() takes
// both of its branches in most warps.
// its constants, formed once on the host: a thread of a launch with one element
// a thread would spend more FP64 time on them than on its element
struct Projection {
    int on;  // 0: copy
    double beta, eta, th, rden;  // th = tanh(beta eta), rden = 1 / (th + tanh(beta (1 - eta)))
};
inline Projection make_projection(int on, double beta, double eta) {
    Projection p{on, beta, eta, 0.0, 1.0};
    if (on) {
        p.th = std::tanh(beta * eta);
        p.rden = 1.0 / (p.th + std::tanh(beta * (1.0 - eta)));
    }
    return p;
}
__device__ __forceinline__ double proj_tanh(double v) {
    const double E = exp(-2.0 * fabs(v));
    return copysign((1.0 - E) / (1.0 + E), v);
}
__device__ __forceinline__ double proj_sech2(double v) {
    const double E = exp(-2.0 * fabs(v)), r = 1.0 / (1.0 + E);
    return 4.0 * E * (r * r);
}
__device__ __forceinline__ double project(const Projection &p, double x) {
    return p.on ? (p.th + proj_tanh(p.beta * (x - p.eta))) * p.rden : x;
}
__device__ __forceinline__ double project_slope(const Projection &p, double x) {
    return p.beta * p.rden * proj_sech2(p.beta * (x - p.eta));
}

}  // namespace topo
