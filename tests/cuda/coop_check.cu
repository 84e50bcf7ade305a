// coop_check.cu -- a wait of the cooperative grid's barrier (coop.cuh) that runs
// out at the kernel's last barrier: one CTA comes late, after another has given up,
// and passes.  The kernel must not report itself as finished, and works again once
// the host has set the counters back.  Prints "barrier OK".
#include <cstdio>

#include "coop.cuh"

using namespace topo;

static __global__ void k_late(GridBar b, int late, int *out, int *status) {
    unsigned arrivals = 0;
    if (!grid_sync(b, arrivals)) return;
    // a delay with an end: 20 ms, where the others wait for about 1
    if ((int)blockIdx.x == late && threadIdx.x == 0)
        for (int i = 0; i < 20000; i++) __nanosleep(1000);
    if (!grid_sync(b, arrivals)) return;
    if (threadIdx.x == 0) out[blockIdx.x] = 1;
    if (grid_leave(b)) {
        *status = 0;
        __threadfence_system();
    }
}

int main() {
    const int CTAS = 8;
    unsigned *c;
    int *out, *status, *status_dev, h[CTAS];
    if (cudaMalloc(&c, 3 * sizeof(unsigned)) || cudaMalloc(&out, sizeof(h)) ||
        cudaHostAlloc((void **)&status, sizeof(int), cudaHostAllocMapped) ||
        cudaHostGetDevicePointer((void **)&status_dev, status, 0) || cudaMemset(c, 0, 12))
        return printf("set-up failed\n"), 1;
    GridBar bar{c, c + 1, c + 2};
    bar.polls = 2000;
    for (int t = 0; t < 4; t++) {  // in time, late, in time, in time
        int late = t == 1 ? CTAS - 1 : -1, done = 0;
        *status = 1;
        cudaMemset(out, 0, sizeof(h));
        void *args[] = {&bar, &late, &out, &status_dev};
        if (cudaLaunchCooperativeKernel((const void *)k_late, dim3(CTAS), dim3(64), args, 0, nullptr) ||
            cudaDeviceSynchronize() || cudaMemcpy(h, out, sizeof(h), cudaMemcpyDeviceToHost))
            return printf("launch %d: %s\n", t, cudaGetErrorString(cudaGetLastError())), 1;
        for (int v : h) done += v;
        if (late < 0 ? (*status != 0 || done != CTAS) : (*status == 0 || done == CTAS))
            return printf("launch %d: status %d with %d of %d CTAs finished\n", t, *status, done, CTAS), 1;
        if (*status) cudaMemset(c, 0, 12);
    }
    unsigned left[3];
    cudaMemcpy(left, c, 12, cudaMemcpyDeviceToHost);
    if (left[0] || left[1] || left[2]) return printf("counters left at %u %u %u\n", left[0], left[1], left[2]), 1;
    printf("barrier OK\n");
    return 0;
}
