// topgpu_streams.h -- streams of the coarsest level's factorisation
#pragma once
#include <cuda_runtime.h>

namespace topgpu {
// The streams and events of factor_and_inverse beside its caller's stream, kept by
// who calls it again and again.
struct FactorStreams {
    cudaStream_t aux = nullptr, inv = nullptr;         // trailing updates; the inverse of the factor
    cudaEvent_t go = nullptr, auxDone = nullptr, invDone = nullptr;
    cudaError_t create()
    {
        cudaError_t e = cudaSuccess;
        for (cudaStream_t *q : {&aux, &inv}) if (!*q && e == cudaSuccess) e = cudaStreamCreateWithFlags(q, cudaStreamNonBlocking);
        for (cudaEvent_t *v : {&go, &auxDone, &invDone}) if (!*v && e == cudaSuccess) e = cudaEventCreateWithFlags(v, cudaEventDisableTiming);
        return e;
    }
    void destroy()
    {
        for (cudaStream_t q : {aux, inv}) if (q) cudaStreamDestroy(q);
        for (cudaEvent_t v : {go, auxDone, invDone}) if (v) cudaEventDestroy(v);
        *this = FactorStreams{};
    }
};
}  // namespace topgpu
