// coop.cuh -- barrier and sums of a cooperative grid.
//
// Iterations whose kernels are shorter than a launch run as one cooperative
// kernel whose CTAs (all resident, cudaLaunchCooperativeKernel) meet at a
// counter in global memory.  Every wait is bounded: a CTA that gives up sets
// `fail`, on which every other CTA that still waits leaves too.  The status of the
// kernel is written by the last CTA to finish (grid_leave), so it is written only
// if none gave up; otherwise the host sets the counters back.
#pragma once
#include <cuda_runtime.h>

namespace topo {

struct GridBar {
    unsigned *count;  // arrivals of this launch; zero between launches
    unsigned *left;   // CTAs that have finished; the last one zeroes both
    unsigned *fail;   // set by a CTA whose wait ran out
    unsigned polls = 1u << 23;  // limit of a wait: some seconds
};

__device__ __forceinline__ unsigned ld_poll(const unsigned *p) {
    unsigned v;
    asm volatile("ld.relaxed.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// every thread of every CTA; `arrivals` counts this CTA's barriers.  False:
// some CTA gave up, and the caller returns at once.
__device__ __forceinline__ bool grid_sync(const GridBar &b, unsigned &arrivals) {
    arrivals++;
    bool ok = true;
    __syncthreads();
    if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(b.count) : "memory");
        const unsigned target = arrivals * gridDim.x;
        unsigned polls = 0;
        while ((int)(ld_poll(b.count) - target) < 0) {  // both may wrap
            if (++polls > b.polls || ((polls & 1023u) == 0 && ld_poll(b.fail))) {
                atomicExch(b.fail, 1u);
                ok = false;
                break;
            }
        }
        __threadfence();
    }
    return __syncthreads_and(ok) != 0;
}

// the end of the kernel, every thread of every CTA: true in one thread of the last
// CTA, once every CTA has come here; counters back to zero for the next launch on
// the same stream
__device__ __forceinline__ bool grid_leave(const GridBar &b) {
    if (threadIdx.x != 0) return false;
    __threadfence();
    if (atomicAdd(b.left, 1u) != gridDim.x - 1) return false;
    *b.count = 0u;
    *b.left = 0u;
    __threadfence();
    return true;
}

// CTA sums of NV FP32 values per thread into out[v * stride], v = 0..NV-1.
// Every thread of the CTA calls it; `sm` is free again after the caller's next
// barrier.
template <int NT, int NV>
__device__ __forceinline__ void cta_sums(const float v[NV], float *sm /* NV * NT / 32 */, float *out, size_t stride) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int i = 0; i < NV; i++) {
        float x = v[i];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        if (lane == 0) sm[i * (NT / 32) + wid] = x;
    }
    __syncthreads();
    if (threadIdx.x < NV) {
        float s = 0.0f;
#pragma unroll
        for (int w = 0; w < NT / 32; w++) s += sm[threadIdx.x * (NT / 32) + w];
        out[threadIdx.x * stride] = s;
    }
}
// The same in FP64.  A scheduler of GB300 issues an FP64 instruction every 64
// clocks, so the additions are spread over the first warps, a value each (one on
// each scheduler for up to four values): NT / 32 + 5 of them in a row instead of
// 5 NV for each of a scheduler's warps and NT / 32 in one thread (MMA update of
// 1769472 variables 1.87 -> 1.84 ms, of 27648 0.212 -> 0.206).  (For the same
// reason scalar FP64 algebra belongs in one thread, not in all.)
template <int NT, int NV>
__device__ __forceinline__ void cta_sums(const double v[NV], double *sm /* NV * NT */, double *out, size_t stride) {
    static_assert(NV <= NT / 32, "a warp per value");
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
    for (int i = 0; i < NV; i++) sm[i * NT + threadIdx.x] = v[i];
    __syncthreads();
    if (wid < NV) {
        const double *p = sm + wid * NT;
        double s = p[lane];
#pragma unroll
        for (int t = 32; t < NT; t += 32) s += p[lane + t];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) out[wid * stride] = s;
    }
}
// after the barrier: the grid's sums of the nv <= NT / 32 values whose CTA sums
// stand at part[v * gridDim + b], the same in every thread of every CTA (a
// fixed order: 32 strided sums, one tree), one warp a value
template <int NT, class V>
__device__ __forceinline__ void grid_totals(const V *part, int nv, V *sm /* nv */) {
    const int lane = threadIdx.x & 31, v = threadIdx.x >> 5;
    if (v < nv) {
        const V *p = part + (size_t)v * gridDim.x;
        V s = V(0);
        // the loads of eight strides in flight at once: one L2 round trip for 256 CTAs
        for (unsigned b = lane; b < gridDim.x; b += 256) {
            V t[8];
#pragma unroll
            for (int u = 0; u < 8; u++) t[u] = b + 32 * u < gridDim.x ? __ldcg(p + b + 32 * u) : V(0);
#pragma unroll
            for (int u = 0; u < 8; u++) s += t[u];
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) sm[v] = s;
    }
    __syncthreads();
}

}  // namespace topo
