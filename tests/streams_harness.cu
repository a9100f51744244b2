// The coarsest level's factorisation and inverse on its streams (topgpu_dense.cuh,
// factor_and_inverse) over symmetric diagonally dominant matrices.  For each size given, with W
// = L^-1 beside the factor and after it: the largest entry of A A^-1 - I, the number
// of W's entries that differ from those of the same kernels on one stream, and of
// those that differ over eight repeats, and the status.
#include <cstdio>
#include <cstdlib>
#include <algorithm>
#include <cmath>
#include <vector>
#include "topgpu_dense.cuh"

using namespace topgpu;
#define CK(x) do { cudaError_t e = (x); if (e != cudaSuccess) { std::printf("CUDA error %s\n", cudaGetErrorString(e)); return 1; } } while (0)

int main(int argc, char **argv)
{
    CK(chol_smem_attr());
    FactorStreams f;
    CK(f.create());
    cudaStream_t st;
    CK(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    for (int a = 1; a < argc; ++a) {
        const int64_t n = std::atoi(argv[a]);
        std::vector<double> A((size_t)(n * n)), X(A.size()), one(A.size()), W(A.size()), R(A.size());
        uint64_t h = 88172645463325252ull + n;
        auto rnd = [&] { h ^= h << 13; h ^= h >> 7; h ^= h << 17; return double(h >> 11) * 0x1p-53 - 0.5; };
        for (int64_t j = 0; j < n; ++j)      // off-diagonal row sums below 1, diagonal in [2, 3]: condition below 4
            for (int64_t i = j; i < n; ++i) A[i + n * j] = A[j + n * i] = i == j ? 2.5 + rnd() : 2.0 * rnd() / double(n);
        double *dA, *dW, *dI, *dR, *D;
        int *ds;
        const size_t b = sizeof(double) * A.size();
        CK(cudaMalloc(&dA, b)); CK(cudaMalloc(&dW, b)); CK(cudaMalloc(&dI, b)); CK(cudaMalloc(&dR, b));
        CK(cudaMalloc(&D, sizeof(double) * kDb * kDb * ((n + kDb - 1) / kDb))); CK(cudaMalloc(&ds, sizeof(int)));
        CK(cudaMemcpy(dR, A.data(), b, cudaMemcpyHostToDevice));
        CK(cudaMemset(ds, 0, sizeof(int)));
        CK(cudaMemcpy(dA, dR, b, cudaMemcpyDeviceToDevice));
        CK(cudaMemset(dW, 0, b));
        for (int64_t k0 = 0; k0 < n; k0 += kPb) {       // one stream, nothing overlaps
            chol_diag_kernel<<<1, kDiagThreads, kDiagSmem>>>(dA, n, k0, D, ds);
            const int64_t rest = n - k0 - kPb;
            if (rest <= 0) break;
            const unsigned nt = (unsigned)((rest + kTileB - 1) / kTileB);
            chol_panel(dA, n, k0, D, 148, 0);
            chol_next(dA, n, k0, 0);
            if (nt > 2) chol_trail_kernel<<<dim3(nt, nt - 2), kTileThreads>>>(dA, n, k0, 2);
        }
        inverse_columns(dA, dW, dI, D, n, 0, n, 0);
        CK(cudaMemcpy(one.data(), dW, b, cudaMemcpyDeviceToHost));
        for (int beside = 1; beside >= 0; --beside) {
            int64_t launches = 0, fromOne = 0, repeats = 0;
            for (int rep = 0; rep < 8; ++rep) {
                CK(cudaMemcpyAsync(dA, dR, b, cudaMemcpyDeviceToDevice, st));
                CK(cudaMemsetAsync(dI, 0xff, b, st));   // NaN: an entry read before it is written shows
                CK(factor_and_inverse(dA, dW, dI, D, n, ds, 148, beside != 0, st, f, launches));
                CK(cudaMemcpyAsync(W.data(), dW, b, cudaMemcpyDeviceToHost, st));
                CK(cudaStreamSynchronize(st));
                if (rep == 0) {
                    R = W;
                    for (size_t i = 0; i < W.size(); ++i) fromOne += !(W[i] == one[i]);
                } else {
                    for (size_t i = 0; i < W.size(); ++i) repeats += !(W[i] == R[i]);
                }
            }
            const unsigned t = (unsigned)((n + kTileB - 1) / kTileB);
            dgemm_tile_kernel<true, true><<<dim3(t, t), kTileThreads, 0, st>>>(dI, n, dW, n, dW, n, (int)n, (int)n, (int)n, 0, 1, 1);
            dgemm_tile_kernel<false, true><<<dim3(t, t), kTileThreads, 0, st>>>(dA, n, dR, n, dI, n, (int)n, (int)n, (int)n, 0, 0, 0);   // A A^-1
            int s = -1;
            CK(cudaMemcpyAsync(X.data(), dA, b, cudaMemcpyDeviceToHost, st));
            CK(cudaMemcpyAsync(&s, ds, sizeof(int), cudaMemcpyDeviceToHost, st));
            CK(cudaStreamSynchronize(st));
            double res = 0;
            for (int64_t j = 0; j < n; ++j)
                for (int64_t i = 0; i < n; ++i) res = std::max(res, std::fabs(X[i + n * j] - (i == j ? 1.0 : 0.0)));
            std::printf("%lld %d %.3e %lld %lld %d\n", (long long)n, beside, res, (long long)fromOne, (long long)repeats, s);
        }
        for (double *q : {dA, dW, dI, dR, D}) CK(cudaFree(q));
        CK(cudaFree(ds));
    }
    f.destroy();
    CK(cudaStreamDestroy(st));
    return 0;
}
