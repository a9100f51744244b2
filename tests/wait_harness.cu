// A column wait of the coarsest factorisation (topgpu_dense.cuh, chol_await) on
// mbarriers that nobody arrives at: prints the status word and the milliseconds of
// one wait by each of two warps, then of 30 more waits a warp.  The waits are
// bounded, so the kernel ends by itself.
#include <cstdio>
#include "topgpu_dense.cuh"

using namespace topgpu;
#define CK(x) do { cudaError_t e = (x); if (e != cudaSuccess) { std::printf("CUDA error %s\n", cudaGetErrorString(e)); return 1; } } while (0)

__global__ void wait_kernel(int waits, int *status)
{
    __shared__ uint64_t ready[32];
    if (threadIdx.x < 32)
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"((unsigned)__cvta_generic_to_shared(ready + threadIdx.x)) : "memory");
    __syncthreads();
    for (int j = 0; j < waits; ++j) chol_await(ready + j, 0, status);
}

int main()
{
    int *st;
    CK(cudaMalloc(&st, sizeof(int)));
    CK(cudaMemset(st, 0, sizeof(int)));
    cudaEvent_t a, b;
    CK(cudaEventCreate(&a));
    CK(cudaEventCreate(&b));
    for (int waits : {1, 30}) {
        int s = -1;
        float ms = 0;
        CK(cudaEventRecord(a));
        wait_kernel<<<1, 64>>>(waits, st);
        CK(cudaEventRecord(b));
        CK(cudaMemcpy(&s, st, sizeof(int), cudaMemcpyDeviceToHost));
        CK(cudaEventElapsedTime(&ms, a, b));
        std::printf("%d %.1f\n", s, ms);
    }
    return 0;
}
