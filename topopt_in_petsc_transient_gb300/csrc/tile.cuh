// tile.cuh -- the matrix-free hex8 operator kernel.
//
// One CTA of 512 threads owns a 7x7x7 brick of output nodes.  It stages the
// 9x9x9 input nodes (brick + one-node halo) in shared memory, lets each thread
// apply the element operator of one of the 8x8x8 elements touching the brick
// (mode-basis form, common.cuh), parks the 24 element outputs in shared memory
// and finally lets each output node gather its 8 element contributions.  No
// atomics: every output is written once, so results are bitwise reproducible.
// Element work on the brick faces is recomputed by the neighbour CTA
// (512/343 = 1.49x redundancy), traded for determinism and zero global
// scatter traffic.
//
// What is staged, how element weights are formed and what happens to the
// assembled value (masking, fused vector updates, dot products) is supplied by
// a policy type; see le.cu for the policies used by the solver.
#pragma once
#include <type_traits>
#include "common.cuh"

namespace topo {

constexpr int TILE = 7;               // output nodes per CTA edge
constexpr int TILE_E = TILE + 1;      // elements per CTA edge
constexpr int TILE_N = TILE + 2;      // staged nodes per CTA edge
constexpr int TILE_THREADS = 512;     // == TILE_E^3
constexpr int TILE_STAGED = TILE_N * TILE_N * TILE_N;  // 729
constexpr int TILE_OUT = TILE * TILE * TILE;            // 343
constexpr int EL_STRIDE = 25;         // padded element-output row (bank spread)
// the same of bricks of TL x TL x TZ output nodes: 7x7x7, in FP64 also 7x7x5 and
// 3x3x3 (launch_brick)
template <int TL, int TZ>
struct TileGeom {
    static constexpr int E = TL + 1, N = TL + 2, THREADS = E * E * (TZ + 1), STAGED = N * N * (TZ + 2);
    static constexpr int OUT = TL * TL * TZ;
    static constexpr int LOG = E == 8 ? 3 : 2;  // E = 2^LOG
    static_assert(E == 1 << LOG && STAGED <= 2 * THREADS, "staging in two passes");
};

template <class T, int TL = TILE, int TZ = TILE>
constexpr size_t tile_smem_bytes() {
    return sizeof(T) * ((size_t)TileGeom<TL, TZ>::STAGED * 3 + (size_t)TileGeom<TL, TZ>::THREADS * EL_STRIDE);
}

__host__ __device__ inline int tile_count(const GridDesc &g, int &ntx, int &nty, int tl = TILE, int tz = TILE) {
    ntx = (g.nx + tl - 1) / tl;
    nty = (g.ny + tl - 1) / tl;
    return ntx * nty * ((g.nz + tz - 1) / tz);
}

// Policy interface:
//   static constexpr bool HAS_K, HAS_M;
//   static constexpr int NRED;     grid-reduced doubles (0..4)
//   __device__ void load(long long n, T v[3]) const;
//   __device__ void coef(long long e, T &ck, T &cm) const;
//   __device__ void epilogue(long long n, int i, int j, int k, const T y[3], double red[]) const;
//   __device__ void finish(const double tot[]) const;   (thread 0 of last CTA)
//   Partials<NRED> part;  (when NRED > 0)
// optional early exit: a policy may define `bool skip() const` (read by every
// thread before any shared-memory or reduction work, so the whole grid exits)
template <class P>
__device__ __forceinline__ auto pol_skip(const P &p, int) -> decltype(p.skip()) {
    return p.skip();
}
template <class P>
__device__ __forceinline__ bool pol_skip(const P &, long) {
    return false;
}

// optional per-thread state read before the first brick: `void begin()`
template <class P>
__device__ __forceinline__ auto pol_begin(P &p, int) -> decltype(p.begin()) {
    p.begin();
}
template <class P>
__device__ __forceinline__ void pol_begin(P &, long) {}

// optional epilogue-operand prefetch: a policy may define `Pre pre(long long n)`
// and `epilogue(n, i, j, k, y, red, const Pre &)`; the kernel issues pre()
// before the element phase so the loads overlap the element arithmetic
struct NoPre {};
template <class P>
__device__ __forceinline__ auto pol_pre(const P &p, long long n, int) -> decltype(p.pre(n)) {
    return p.pre(n);
}
template <class P>
__device__ __forceinline__ NoPre pol_pre(const P &, long long, long) {
    return NoPre{};
}
template <class P, class T, class A, class R>
__device__ __forceinline__ auto pol_epi(const P &p, long long n, int i, int j, int k, const T y[3], A *red,
                                        const R &pre, int) -> decltype(p.epilogue(n, i, j, k, y, red, pre)) {
    return p.epilogue(n, i, j, k, y, red, pre);
}
template <class P, class T, class A, class R>
__device__ __forceinline__ void pol_epi(const P &p, long long n, int i, int j, int k, const T y[3], A *red,
                                        const R &, long) {
    p.epilogue(n, i, j, k, y, red);
}

// per-thread accumulator type of a policy's reductions: `using Red = float;`
// in an FP32 policy keeps the per-node sums on the FP32 pipe (GB300 runs FP64
// at 1/64 of the FP32 rate); the thread's partials widen to FP64 once, for the
// grid reduction
template <class P, class = void>
struct pol_red {
    using type = double;
};
template <class P>
struct pol_red<P, std::void_t<typename P::Red>> {
    using type = typename P::Red;
};
template <class P>
using pol_red_t = typename pol_red<P>::type;

// position of a brick in the grid of bricks.  The persistent kernels step it by
// the grid size without dividing again: three quotients by run-time numbers, per
// thread and brick, were a tenth of the FP32 product's instructions
struct TilePos {
    int i, j, k;
};
__device__ __forceinline__ TilePos tile_pos(int tile, int ntx, int nty) {
    const int q = tile / ntx, k = q / nty;
    return {tile - q * ntx, q - k * nty, k};
}
__device__ __forceinline__ TilePos tile_next(TilePos p, TilePos step, int ntx, int nty) {
    p.i += step.i;
    p.j += step.j + (p.i >= ntx);
    p.i -= p.i >= ntx ? ntx : 0;
    p.k += step.k + (p.j >= nty);
    p.j -= p.j >= nty ? nty : 0;
    return p;
}

// index arithmetic of the kernels in 32 bits (a node index fits, lex3): unsigned
// comparisons, and widened once for the addresses
__device__ __forceinline__ bool tile_in(int i, int j, int k, int nx, int ny, int nz) {
    return (unsigned)i < (unsigned)nx && (unsigned)j < (unsigned)ny && (unsigned)k < (unsigned)nz;
}
__device__ __forceinline__ long long tile_index(int i, int j, int k, int nx, int ny) {
    return (unsigned)i + (unsigned)nx * ((unsigned)j + (unsigned)ny * (unsigned)k);
}

// staged input nodes of a brick held by this thread (at most two)
template <class T, int TL = TILE, int TZ = TILE, class Pol>
__device__ __forceinline__ void tile_fetch(const Pol &pol, const GridDesc &g, TilePos at, T v[2][3]) {
    using G = TileGeom<TL, TZ>;
    const int i0 = at.i * TL, j0 = at.j * TL, k0 = at.k * TZ;
#pragma unroll
    for (int it = 0; it < 2; it++) {
        const int s = threadIdx.x + it * G::THREADS;
        const int lx = s % G::N, ly = (s / G::N) % G::N, lz = s / (G::N * G::N);
        const int gi = i0 - 1 + lx, gj = j0 - 1 + ly, gk = k0 - 1 + lz;
        if (s < G::STAGED && tile_in(gi, gj, gk, g.nx, g.ny, g.nz)) {
            const long long n = tile_index(gi, gj, gk, g.nx, g.ny);
            pol.load(n, v[it]);
        } else {
            v[it][0] = v[it][1] = v[it][2] = T(0);
        }
    }
}

// ---------------------------------------------------------------------------
// element phase and gather, shared by both staging paths
// ---------------------------------------------------------------------------
// one element per thread: the 24 outputs of element (lx, ly, lz) of the brick
// at (i0, j0, k0) from the staged nodes sIn into sEl
template <class T, int TL = TILE, int TZ = TILE, class Pol>
__device__ __forceinline__ void tile_elements(const GridDesc &g, const ElemConst<T> &C, const Pol &pol, const T *sIn,
                                              T *sEl, int i0, int j0, int k0) {
    using G = TileGeom<TL, TZ>;
    const int tid = threadIdx.x;
    const int lx = tid & (G::E - 1), ly = (tid >> G::LOG) & (G::E - 1), lz = tid >> (2 * G::LOG);
    const int ei = i0 - 1 + lx, ej = j0 - 1 + ly, ek = k0 - 1 + lz;
    T *out = sEl + tid * EL_STRIDE;
    if (tile_in(ei, ej, ek, g.ex, g.ey, g.ez)) {
        const long long e = tile_index(ei, ej, ek, g.ex, g.ey);
        T ck, cm;
        pol.coef(e, ck, cm);
        T U[3][8];
#pragma unroll
        for (int L = 0; L < 8; L++) {
            int s = (lx + (L & 1)) + G::N * ((ly + ((L >> 1) & 1)) + G::N * (lz + (L >> 2)));
#pragma unroll
            for (int c = 0; c < 3; c++) U[c][L] = sIn[s * 3 + c];
        }
#pragma unroll
        for (int c = 0; c < 3; c++) mode_fwd(U[c]);
        T Y[3][8];
        if (Pol::HAS_K) {
            mode_khat_mass<Pol::HAS_M>(C, ck, cm, U, Y);
        } else {
#pragma unroll
            for (int b = 0; b < 3; b++)
#pragma unroll
                for (int m = 0; m < 8; m++) Y[b][m] = tadd(T(0), tmul(tmul(cm, C.W[m]), U[b][m]));
        }
#pragma unroll
        for (int b = 0; b < 3; b++) {
            mode_bwd(Y[b]);
#pragma unroll
            for (int L = 0; L < 8; L++) out[L * 3 + b] = Y[b][L];
        }
    } else {
#pragma unroll
        for (int q = 0; q < 24; q++) out[q] = T(0);
    }
}

// the output node (tx, ty, tz) of this thread: its 8 element contributions
// from sEl, then the policy epilogue
template <class T, int TL = TILE, int TZ = TILE, class Pol, class R>
__device__ __forceinline__ void tile_gather(const Pol &pol, const T *sEl, long long on, int oi, int oj, int ok, int tx,
                                            int ty, int tz, const R &pre, pol_red_t<Pol> *red) {
    constexpr int E = TileGeom<TL, TZ>::E;
    T y[3] = {T(0), T(0), T(0)};
#pragma unroll
    for (int L = 0; L < 8; L++) {
        int ax = L & 1, ay = (L >> 1) & 1, az = L >> 2;
        int le = (tx + 1 - ax) + E * ((ty + 1 - ay) + E * (tz + 1 - az));
#pragma unroll
        for (int c = 0; c < 3; c++) y[c] = tadd(y[c], sEl[le * EL_STRIDE + L * 3 + c]);
    }
    pol_epi(pol, on, oi, oj, ok, y, red, pre, 0);
}

// ---------------------------------------------------------------------------
// staging path 1: per-thread loads into registers
// ---------------------------------------------------------------------------
// FP32 kernels are persistent: the grid holds as many CTAs as fit on the
// device, each CTA walks the bricks tile = blockIdx.x, + gridDim.x, ... and
// loads the next brick's staged nodes into registers while it computes the
// current one, so the global-load latency of the staging overlaps the element
// arithmetic.  Reductions accumulate over a CTA's bricks in a fixed order and
// are reduced once over the grid.  FP64 and double-float kernels (one CTA of
// 128 registers a thread per SM) cannot hold the next brick's values: they
// prefetch into shared memory instead (staging path 2) when their policy
// allows it, and otherwise launch one CTA per brick.
template <class T>
constexpr bool tile_persistent() {
    return sizeof(T) == 4;
}
// Two barriers a brick: the staged nodes are free once the element phase is over,
// so the next brick is staged beside the gather, and the element outputs once every
// thread has come to the next staging barrier.
// one brick: stage (v holds its staged nodes), element phase, gather and
// epilogue; with `more` the staged nodes of brick `next` are loaded into v while
// this brick is computed
template <class T, int TL = TILE, int TZ = TILE, class Pol>
__device__ __forceinline__ void tile_brick(const GridDesc &g, const ElemConst<T> &C, const Pol &pol, T *sIn, T *sEl,
                                           TilePos at, TilePos next, bool more, T v[2][3],
                                           pol_red_t<Pol> *red) {
    using G = TileGeom<TL, TZ>;
    const int tid = threadIdx.x;
    const int i0 = at.i * TL, j0 = at.j * TL, k0 = at.k * TZ;
#pragma unroll
    for (int it = 0; it < 2; it++) {
        const int s = tid + it * G::THREADS;
        if (s < G::STAGED) {
#pragma unroll
            for (int c = 0; c < 3; c++) sIn[s * 3 + c] = v[it][c];
        }
    }
    // output node of this thread and its prefetched epilogue operands
    const int tx = tid % TL, ty = (tid / TL) % TL, tz = tid / (TL * TL);
    const int oi = i0 + tx, oj = j0 + ty, ok = k0 + tz;
    const bool has_out = tid < G::OUT && oi < g.nx && oj < g.ny && ok < g.nz;
    const long long on = has_out ? tile_index(oi, oj, ok, g.nx, g.ny) : 0;
    const auto pre = pol_pre(pol, on, 0);
    __syncthreads();
    if (more) tile_fetch<T, TL, TZ>(pol, g, next, v);
    tile_elements<T, TL, TZ>(g, C, pol, sIn, sEl, i0, j0, k0);
    __syncthreads();
    if (has_out) tile_gather<T, TL, TZ>(pol, sEl, on, oi, oj, ok, tx, ty, tz, pre, red);
}

// ---------------------------------------------------------------------------
// staging path 2: per-thread asynchronous copies into shared memory
// ---------------------------------------------------------------------------
// For kernels whose registers are all taken by the element arithmetic (FP64
// and double-float, one CTA of 512 threads per SM) the next brick cannot be
// held in registers.  A policy may then opt in to this path by declaring
//   using Src = float | double;          element type of its raw input arrays
//   static constexpr int NSRC;           raw arrays staged per node (1 or 2)
//   static constexpr bool MASK;          read the clamp bitmask `fixed` too
//   const Src *src(int k) const;         raw array k, 3 values per node
//   void xform(const Src raw[NSRC][3], uint8_t f, T v[3]) const;
//                                        staged value from the raw values
// The kernel is then persistent: every thread issues `cp.async` copies of the
// raw values of its own staged nodes of the next brick into its own slots of a
// raw buffer in shared memory (and a plain load of their mask bytes into
// registers) while the current brick is computed, and converts them into the
// staged nodes after waiting for its own copies only.  No register holds the
// prefetched brick, and no barrier guards the raw buffer: each slot is written
// and read by one thread.
//
// (A bulk-copy form, one `cp.async.bulk` per 16-byte-aligned node row of the
// staged brick completing on an mbarrier, was measured slower: 162 to 243
// copies of 32 to 224 bytes per brick keep the copy engine busy for about 28
// cycles each, and the FP32 product took 219 instead of 98 us at 192x96x96.
// The node rows (3 nx values) are not 16-byte multiples, so no tensor map
// describes the bricks.)
template <class P, class = void>
struct pol_async : std::false_type {};
template <class P>
struct pol_async<P, std::void_t<typename P::Src>> : std::true_type {};

// the async path serves the non-persistent (FP64, double-float) kernels; FP32
// kernels keep their register prefetch
template <class T, class Pol>
constexpr bool tile_async() {
    return pol_async<Pol>::value && !tile_persistent<T>();
}

template <class T, class Pol, bool ASYNC = tile_async<T, Pol>()>
struct TileSmem {
    static constexpr size_t bytes = tile_smem_bytes<T>();
};
template <class T, class Pol>
struct TileSmem<T, Pol, true> {
    using Src = typename Pol::Src;
    static constexpr size_t raw = 0;  // [NSRC][TILE_STAGED][3] Src
    static constexpr size_t in = ((size_t)Pol::NSRC * TILE_STAGED * 3 * sizeof(Src) + 15) / 16 * 16;
    static constexpr size_t el = in + sizeof(T) * (size_t)TILE_STAGED * 3;
    static constexpr size_t bytes = el + sizeof(T) * (size_t)TILE_THREADS * EL_STRIDE;
};

template <int NB>
__device__ __forceinline__ void cp_async(void *dst, const void *src) {
    static_assert(NB == 4 || NB == 8, "cp.async of one FP32 or FP64 value");
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src),
                 "n"(NB)
                 : "memory");
}

// this thread's staged nodes of a brick: raw values by cp.async into its
// slots of `raw`, mask bytes into f
template <class T, class Pol>
__device__ __forceinline__ void tile_fetch_async(const Pol &pol, const GridDesc &g, TilePos at,
                                                 typename Pol::Src *raw, uint8_t f[2]) {
    using Src = typename Pol::Src;
    const int i0 = at.i * TILE, j0 = at.j * TILE, k0 = at.k * TILE;
#pragma unroll
    for (int it = 0; it < 2; it++) {
        const int s = threadIdx.x + it * TILE_THREADS;
        const int lx = s % TILE_N, ly = (s / TILE_N) % TILE_N, lz = s / (TILE_N * TILE_N);
        const int gi = i0 - 1 + lx, gj = j0 - 1 + ly, gk = k0 - 1 + lz;
        f[it] = 0;
        if (s < TILE_STAGED && tile_in(gi, gj, gk, g.nx, g.ny, g.nz)) {
            const long long n = tile_index(gi, gj, gk, g.nx, g.ny);
#pragma unroll
            for (int k = 0; k < Pol::NSRC; k++)
#pragma unroll
                for (int c = 0; c < 3; c++)
                    cp_async<(int)sizeof(Src)>(raw + ((size_t)k * TILE_STAGED + s) * 3 + c, pol.src(k) + 3 * n + c);
            if constexpr (Pol::MASK) f[it] = pol.fixed[n];
        }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
}

template <class T, class Pol>
__device__ __forceinline__ void tile_run_async(const GridDesc &g, const ElemConst<T> &C, const Pol &pol,
                                               unsigned char *sm, int ntiles, int ntx, int nty, pol_red_t<Pol> *red) {
    using L = TileSmem<T, Pol>;
    using Src = typename Pol::Src;
    const int tid = threadIdx.x;
    Src *raw = reinterpret_cast<Src *>(sm + L::raw);
    T *sIn = reinterpret_cast<T *>(sm + L::in);
    T *sEl = reinterpret_cast<T *>(sm + L::el);
    uint8_t f[2];
    TilePos at = tile_pos(blockIdx.x, ntx, nty);
    const TilePos step = tile_pos(gridDim.x, ntx, nty);
    if ((int)blockIdx.x < ntiles) tile_fetch_async<T>(pol, g, at, raw, f);
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const TilePos next = tile_next(at, step, ntx, nty);
        const int i0 = at.i * TILE, j0 = at.j * TILE, k0 = at.k * TILE;
        at = next;
        asm volatile("cp.async.wait_group 0;" ::: "memory");  // this thread's copies only
        // raw values -> staged nodes (zero outside the domain)
#pragma unroll
        for (int it = 0; it < 2; it++) {
            const int s = tid + it * TILE_THREADS;
            if (s < TILE_STAGED) {
                const int lx = s % TILE_N, ly = (s / TILE_N) % TILE_N, lz = s / (TILE_N * TILE_N);
                const int gi = i0 - 1 + lx, gj = j0 - 1 + ly, gk = k0 - 1 + lz;
                T v[3] = {T(0), T(0), T(0)};
                if (tile_in(gi, gj, gk, g.nx, g.ny, g.nz)) {
                    Src rv[Pol::NSRC][3];
#pragma unroll
                    for (int k = 0; k < Pol::NSRC; k++)
#pragma unroll
                        for (int c = 0; c < 3; c++) rv[k][c] = raw[((size_t)k * TILE_STAGED + s) * 3 + c];
                    pol.xform(rv, f[it], v);
                }
#pragma unroll
                for (int c = 0; c < 3; c++) sIn[s * 3 + c] = v[c];
            }
        }
        const int tx = tid % TILE, ty = (tid / TILE) % TILE, tz = tid / (TILE * TILE);
        const int oi = i0 + tx, oj = j0 + ty, ok = k0 + tz;
        const bool has_out = tid < TILE_OUT && oi < g.nx && oj < g.ny && ok < g.nz;
        const long long on = has_out ? tile_index(oi, oj, ok, g.nx, g.ny) : 0;
        const auto pre = pol_pre(pol, on, 0);
        __syncthreads();
        if (tile + (int)gridDim.x < ntiles) tile_fetch_async<T>(pol, g, next, raw, f);
        tile_elements<T>(g, C, pol, sIn, sEl, i0, j0, k0);
        __syncthreads();
        if (has_out) tile_gather<T>(pol, sEl, on, oi, oj, ok, tx, ty, tz, pre, red);
    }
}

template <class T, class Pol, int TL = TILE, int TZ = TILE>
__global__ void __launch_bounds__(TileGeom<TL, TZ>::THREADS, sizeof(T) == 4 ? 2 : 1) k_tile(const GridDesc g, const ElemConst<T> C, Pol pol) {
    grid_dep_wait();
    TOPO_DYNAMIC_SMEM(unsigned char, smem_raw);
    if (pol_skip(pol, 0)) return;
    pol_begin(pol, 0);
    int ntx, nty;
    const int ntiles = tile_count(g, ntx, nty, TL, TZ);
    pol_red_t<Pol> red[Pol::NRED > 0 ? Pol::NRED : 1];
#pragma unroll
    for (int r = 0; r < (Pol::NRED > 0 ? Pol::NRED : 1); r++) red[r] = 0;
    static_assert((TL == TILE && TZ == TILE) || !(tile_async<T, Pol>() || tile_persistent<T>()), "other bricks: one a CTA");
    if constexpr (tile_async<T, Pol>()) {
        tile_run_async<T>(g, C, pol, smem_raw, ntiles, ntx, nty, red);
    } else {
        T *sIn = reinterpret_cast<T *>(smem_raw);
        T *sEl = sIn + TileGeom<TL, TZ>::STAGED * 3;
        T v[2][3];
        TilePos at = tile_pos(blockIdx.x, ntx, nty);
        if constexpr (tile_persistent<T>()) {
            const TilePos step = tile_pos(gridDim.x, ntx, nty);
            if ((int)blockIdx.x < ntiles) tile_fetch<T, TL, TZ>(pol, g, at, v);
            for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
                const TilePos next = tile_next(at, step, ntx, nty);
                tile_brick<T, TL, TZ>(g, C, pol, sIn, sEl, at, next, tile + (int)gridDim.x < ntiles, v, red);
                at = next;
            }
        } else {
            tile_fetch<T, TL, TZ>(pol, g, at, v);
            tile_brick<T, TL, TZ>(g, C, pol, sIn, sEl, at, at, false, v, red);
        }
    }
    if constexpr (Pol::NRED > 0) {
        double tot[Pol::NRED];
        if (grid_reduce<TileGeom<TL, TZ>::THREADS, Pol::NRED>(red, pol.part, tot)) pol.finish(tot);
    }
}

}  // namespace topo
