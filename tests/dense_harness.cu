// Runs the coarsest level's dense kernels (topgpu_dense.cuh) on symmetric
// diagonally dominant matrices of the sizes given and prints, per size, the
// largest entry of A A^-1 - I, the largest difference between A^-1 and its
// transpose, and the status flag.  sms=N among the arguments sets the number of SMs
// that the panel's rule reckons with for the sizes after it, neg=R makes the
// diagonal entry of row R negative.
#include <cstdio>
#include <cstdlib>
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>
#include "topgpu_dense.cuh"

using namespace topgpu;
#define CK(x) do { cudaError_t e = (x); if (e != cudaSuccess) { std::printf("CUDA error %s\n", cudaGetErrorString(e)); return 1; } } while (0)

int main(int argc, char **argv)
{
    CK(chol_smem_attr());
    int sms = 148, neg = -1;
    for (int a = 1; a < argc; ++a) {
        if (!std::strncmp(argv[a], "sms=", 4)) { sms = std::atoi(argv[a] + 4); continue; }
        if (!std::strncmp(argv[a], "neg=", 4)) { neg = std::atoi(argv[a] + 4); continue; }
        const int64_t n = std::atoi(argv[a]);
        std::vector<double> A((size_t)(n * n)), X(A.size());
        uint64_t h = 88172645463325252ull + n;
        auto rnd = [&] { h ^= h << 13; h ^= h >> 7; h ^= h << 17; return double(h >> 11) * 0x1p-53 - 0.5; };
        for (int64_t j = 0; j < n; ++j)      // off-diagonal row sums below 1, diagonal in [2, 3]: condition below 4
            for (int64_t i = j; i < n; ++i) A[i + n * j] = A[j + n * i] = i == j ? 2.5 + rnd() : 2.0 * rnd() / double(n);
        if (neg >= 0 && neg < n) A[neg + n * neg] = -1.0;
        double *dA, *W, *I, *D;
        int *st;
        const size_t b = sizeof(double) * A.size();
        CK(cudaMalloc(&dA, b)); CK(cudaMalloc(&W, b)); CK(cudaMalloc(&I, b));
        CK(cudaMalloc(&D, sizeof(double) * kDb * kDb * ((n + kDb - 1) / kDb))); CK(cudaMalloc(&st, sizeof(int)));
        CK(cudaMemset(st, 0, sizeof(int))); CK(cudaMemset(W, 0, b));
        CK(cudaMemcpy(dA, A.data(), b, cudaMemcpyHostToDevice));
        for (int64_t k0 = 0; k0 < n; k0 += kPb) {
            chol_diag_kernel<<<1, kDiagThreads, kDiagSmem>>>(dA, n, k0, D, st);
            const int64_t rest = n - k0 - kPb;
            if (rest > 0) {
                const unsigned nt = (unsigned)((rest + kTileB - 1) / kTileB);
                chol_panel(dA, n, k0, D, sms, 0);
                chol_next(dA, n, k0, 0);
                if (nt > 2) chol_trail_kernel<<<dim3(nt, nt - 2), kTileThreads>>>(dA, n, k0, 2);
            }
            if (sms != 12) inverse_columns(dA, W, I, D, n, k0, std::min<int64_t>(n, k0 + kPb), 0);
        }
        if (sms == 12) inverse_columns(dA, W, I, D, n, 0, n, 0);       // both orders of the inversion
        const unsigned t = (unsigned)((n + kTileB - 1) / kTileB);
        dgemm_tile_kernel<true, true><<<dim3(t, t), kTileThreads>>>(I, n, W, n, W, n, (int)n, (int)n, (int)n, 0, 1, 1);
        int s = -1;
        CK(cudaMemcpy(X.data(), I, b, cudaMemcpyDeviceToHost)); CK(cudaMemcpy(&s, st, sizeof(int), cudaMemcpyDeviceToHost));
        double res = 0, asym = 0;
        for (int64_t j = 0; j < n; ++j)
            for (int64_t i = 0; i < n; ++i) {
                long double v = i == j ? -1.0L : 0.0L;
                for (int64_t k = 0; k < n; ++k) v += (long double)A[k + n * i] * X[k + n * j];
                res = std::max(res, (double)fabsl(v));
                asym = std::max(asym, std::fabs(X[i + n * j] - X[j + n * i]));
            }
        std::printf("%lld %.3e %.3e %d\n", (long long)n, res, asym, s);
        CK(cudaFree(dA)); CK(cudaFree(W)); CK(cudaFree(I)); CK(cudaFree(D)); CK(cudaFree(st));
    }
    return 0;
}
