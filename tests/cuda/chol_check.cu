// chol_check.cu -- the panels of the coarse Cholesky factorisation taken one
// after the other by a single warp, the diagonal block's first and last: blocks
// of a launch run in any order, so both have to give the same factor to the bit.
// Then the inverse from it against the matrix.  Prints "cholesky OK".
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "kernels.cuh"

using namespace topo;

static __global__ void k_panel_in_order(double *A, int n, int k0, double *U, double *Q, int nb, int last_first) {
    for (int t = 0; t < nb; t++) {
        chol_panel(A, n, k0, U, Q, last_first ? nb - 1 - t : t);
        __syncwarp();
    }
}

int main() {
    for (int n : {1, 31, 32, 33, 100, 675}) {
        const size_t nn = (size_t)n * n;
        std::vector<double> G(nn), A(nn);
        unsigned long long x = 88172645463325252ull;
        for (double &g : G) {
            x ^= x << 13, x ^= x >> 7, x ^= x << 17;
            g = (double)(x >> 11) / 9007199254740992.0 - 0.5;
        }
        for (int i = 0; i < n; i++)
            for (int j = 0; j < n; j++) {
                double s = i == j ? 0.1 * n : 0.0;
                for (int k = 0; k < n; k++) s += G[(size_t)i * n + k] * G[(size_t)j * n + k];
                A[(size_t)i * n + j] = s;
            }
        double *dA, *dW, *dU;
        float *df;
        if (cudaMalloc(&dA, 8 * nn) || cudaMalloc(&dW, 8 * nn) || cudaMalloc(&dU, 16 * (size_t)CH * n) ||
            cudaMalloc(&df, 4 * nn))
            return printf("allocation failed\n"), 1;
        std::vector<double> L[2], U[2];
        for (int o = 0; o < 2; o++) {
            L[o].resize(nn);
            U[o].resize(2 * (size_t)CH * n);
            cudaMemcpy(dA, A.data(), 8 * nn, cudaMemcpyHostToDevice);
            cudaMemset(dU, 0, 16 * (size_t)CH * n);
            k_panel_in_order<<<1, 32>>>(dA, n, 0, dU, dU + (size_t)CH * n, (n + CH - 1) / CH, o);
            cudaMemcpy(L[o].data(), dA, 8 * nn, cudaMemcpyDeviceToHost);
            if (cudaMemcpy(U[o].data(), dU, 16 * (size_t)CH * n, cudaMemcpyDeviceToHost)) return printf("failed\n"), 1;
        }
        if (memcmp(L[0].data(), L[1].data(), 8 * nn) || memcmp(U[0].data(), U[1].data(), 16 * (size_t)CH * n))
            return printf("n = %d: the factor depends on the order of the blocks\n", n), 1;
        cudaMemcpy(dA, A.data(), 8 * nn, cudaMemcpyHostToDevice);
        chol_inverse(dA, df, n, dW, dU, nullptr);
        std::vector<double> B(nn);
        if (cudaMemcpy(B.data(), dA, 8 * nn, cudaMemcpyDeviceToHost)) return printf("failed\n"), 1;
        // condition number below 10: A B - I within 1e-12 for sums of up to 675 terms
        double worst = 0.0;
        for (int i = 0; i < n; i++)
            for (int j = 0; j < n; j++) {
                double s = i == j ? -1.0 : 0.0;
                for (int k = 0; k < n; k++) s += A[(size_t)i * n + k] * B[(size_t)k * n + j];
                worst = fmax(worst, fabs(s));
            }
        if (!(worst < 1e-12)) return printf("n = %d: A inv(A) - I = %g\n", n, worst), 1;
        cudaFree(dA), cudaFree(dW), cudaFree(dU), cudaFree(df);
    }
    printf("cholesky OK\n");
    return 0;
}
