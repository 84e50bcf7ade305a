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

// Smoothed Heaviside projection (Filter.h:80-88),
//   (tanh(beta eta) + tanh(beta (x - eta))) / (tanh(beta eta) + tanh(beta (1 - eta))),
// with one exponential and one quotient: tanh v = -+m / (2 + m), m = exp(-2 |v|) - 1.
// FP64 runs at 2 lanes a clock and SM here, and tanh() takes both of its branches in
// most warps (PDE filter at 192x96x96 2.64 instead of 2.59 ms).  Where tanh(beta eta)
// is under a half (small beta or eta) the sum can be small against rounding of E
// near 1, and m is expm1's (density filter at 96x48x48 252 instead of 245 us).
// The ends are fixed and not left to rounding: 0 and 1 go to 0 and 1, and a density
// between them stays between them (one below 0 makes x^p NaN).
// constants, formed once on the host: a thread of a launch with one element a
// thread would spend more FP64 time on them than on its element
struct Projection {
    int on, small;  // on = 0: copy; small: tanh(beta eta) under a half
    double beta, eta, th, rden;  // th = tanh(beta eta), rden = 1 / (th + tanh(beta (1 - eta)))
    double lo, hi;               // 0 and 1 (beta = 0, which has no projection: not a number)
};
inline Projection make_projection(int on, double beta, double eta) {
    Projection p{on, 0, beta, eta, 0.0, 1.0, 0.0, 1.0};
    if (on) {
        p.th = std::tanh(beta * eta);
        p.small = !(p.th >= 0.5);
        p.rden = 1.0 / (p.th + std::tanh(beta * (1.0 - eta)));
        p.lo = 0.0 * p.rden;
        p.hi = 1.0 + p.lo;
    }
    return p;
}
__device__ __forceinline__ double project(const Projection &p, double x) {
    if (!p.on) return x;
    const double v = p.beta * (x - p.eta), w = -2.0 * fabs(v), m = p.small ? expm1(w) : exp(w) - 1.0, q = 2.0 + m;
    const double y = fma(p.th, q, copysign(m, v)) / q * p.rden;
    // on the integer pipes: the bits of a double order like its magnitude, and those
    // above infinity's are not a number
    const long long bx = __double_as_longlong(x), by = __double_as_longlong(y), one = 0x3FF0000000000000ll;
    const bool under = by < 0 && (unsigned long long)by <= 0xFFF0000000000000ull;
    const bool over = by > one && by <= 0x7FF0000000000000ll;
    if (bx << 1 == 0) return p.lo;
    if (bx == one) return p.hi;
    return under && bx >= 0 ? 0.0 : (over && bx < one ? 1.0 : y);
}
// 1 - tanh^2 v = 4 E / (1 + E)^2, E = exp(-2 |v|)
__device__ __forceinline__ double project_slope(const Projection &p, double x) {
    const double E = exp(-2.0 * fabs(p.beta * (x - p.eta))), r = 1.0 / (1.0 + E);
    return p.beta * p.rden * (4.0 * E * (r * r));
}

}  // namespace topo
