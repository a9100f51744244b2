// topgpu_dropin.cu -- the six MEX kernels of TOP_GPU as C-ABI entry points
// for sm_100a.  Same arguments, layouts and in-place semantics as the MEX
// gateways (see include/topgpu.h for the file:line each one replaces).
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>
#include <mutex>
#include "topgpu_kernels.cuh"

using namespace topgpu;

namespace {

inline cudaStream_t S(void *s) { return reinterpret_cast<cudaStream_t>(s); }

// ---------------------------------------------------------------------------
// gather: one thread per element; node ids held in registers; 24 coalesced
// column stores (uMat is column-major [nElem x 24]).  An out-of-range node
// id yields 0 instead of an out-of-bounds read.
template <typename T, typename IDX>
__global__ void gather_kernel(T *__restrict__ uMat, const T *__restrict__ u,
                              const IDX *__restrict__ eNod, int64_t nElem, int64_t nNodes)
{
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nElem) return;
    int64_t node[8];
#pragma unroll
    for (int n = 0; n < 8; ++n) node[n] = (int64_t)__ldg(&eNod[e + n * nElem]) - 1;
#pragma unroll
    for (int n = 0; n < 8; ++n) {
        const bool ok = node[n] >= 0 && node[n] < nNodes;
#pragma unroll
        for (int c = 0; c < 3; ++c)
            uMat[e + (int64_t)(3 * n + c) * nElem] = ok ? __ldg(&u[node[n] + c * nNodes]) : T(0);
    }
}

// scatter: one thread per element; its contributions are fire-and-forget
// reductions into the L2-resident node array, whose rate bounds the kernel.
// Elements that follow one another in y are neighbouring lanes, and the four nodes of
// a's upper face are the four of the next one's lower face (corners 0, 1, 4, 5 and
// 3, 2, 7, 6): where the ids say so, whatever the numbering, the next lane
// adds the value to its own first, which leaves 12 reductions an element of 24
// (524,288 elements in double, gather and scatter and the clear between: 80 -> 74 us, the
// scatter 23 of them; its 117 MB take 18 at the measured copy rate).  Sums of pairs round
// no further off: 9.1e-17 against 1.04e-16 rms over eight values one by one.
template <typename T>
__global__ void scatter_kernel(T *__restrict__ Y, const int32_t *__restrict__ eNod,
                               const T *__restrict__ uMat, int64_t Ne, int64_t nNodes)
{
    const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int lane = threadIdx.x & 31;
    const bool in = e < Ne;
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        constexpr int up[4] = {0, 1, 4, 5}, low[4] = {3, 2, 7, 6};
        int64_t hi = -1, lo = -1;
        T vh[3] = {}, vl[3] = {};
        if (in) {
            hi = (int64_t)__ldg(&eNod[e + up[p] * Ne]) - 1;
            lo = (int64_t)__ldg(&eNod[e + low[p] * Ne]) - 1;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                vh[c] = __ldg(&uMat[e + (int64_t)(c + 3 * up[p]) * Ne]);
                vl[c] = __ldg(&uMat[e + (int64_t)(c + 3 * low[p]) * Ne]);
            }
            if (hi >= nNodes) hi = -1;               // ids out of range add nothing
            if (lo >= nNodes) lo = -1;
        }
        const bool given = __shfl_down_sync(0xffffffffu, lo, 1) == hi && lane < 31;       // the next lane takes it
        const bool taken = __shfl_up_sync(0xffffffffu, hi, 1) == lo && lane > 0;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const T v = __shfl_up_sync(0xffffffffu, vh[c], 1);
            if (taken) vl[c] += v;
            if (lo >= 0) atomicAdd(&Y[lo + c * nNodes], vl[c]);
            if (hi >= 0 && !given) atomicAdd(&Y[hi + c * nNodes], vh[c]);
        }
    }
}

template <typename T>
__global__ void scatter_accum3_kernel(const int32_t *__restrict__ keys, const T *__restrict__ Tmp,
                                      int64_t N, T *__restrict__ xF, int64_t M)
{
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N) return;
    const int64_t key = (int64_t)__ldg(&keys[i]) - 1;
    if (key < 0 || key >= M) return;
#pragma unroll
    for (int c = 0; c < 3; ++c) atomicAdd(&xF[key + c * M], __ldg(&Tmp[i + c * N]));
}

// the element matrix of every regular child, before its modulus
template <typename T>
struct K0Child {
    const T *K0;
    __device__ double operator()(int32_t, int i) const { return double(K0[i]); }
};
struct NoSkip { __device__ bool operator()(int32_t) const { return false; } };

// A row of the level-2 GEMM: the moduli of a coarse cell's regular children
// (0 for void children and for children with fixed DOFs).
template <typename T>
struct Level2Row {
    const int32_t *upMap; const T *E; const int32_t *mapUnique; int64_t nElem; int nCh; int hasFixed;
    __device__ int32_t child(int64_t m, int k) const { return k < nCh ? upMap[m + (int64_t)k * nElem] : 0; }
    __device__ double value(int32_t f0) const { return double(E[f0]); }
    __device__ bool regular(int32_t f0) const { return !(hasFixed && mapUnique[f0] > 0); }
};

template <typename T>
struct Level2Child {   // K_child of assembleKs_level2_inplace.cu:104-115
    const T *E; const T *K0; const int32_t *mapUnique; const T *uFree; const T *uFixed; int hasFixed;
    __device__ double operator()(int32_t f0, int i) const {
        const double mod = double(E[f0]);
        const int32_t uid0 = hasFixed ? mapUnique[f0] - 1 : -1;
        if (uid0 >= 0) return double(uFree[(size_t)uid0 * 576 + i]) * mod + double(uFixed[(size_t)uid0 * 576 + i]);
        return double(K0[i]) * mod;
    }
};
struct RegularChild {  // skip children with fixed DOFs (handled by the GEMM otherwise)
    const int32_t *mapUnique; int hasFixed; int invert;
    __device__ bool operator()(int32_t f0) const {
        const bool bnd = hasFixed && mapUnique[f0] > 0;
        return invert ? !bnd : bnd;
    }
};
template <typename T>
struct PrevChild {
    const T *KsPrev;
    __device__ double operator()(int32_t f0, int i) const { return double(KsPrev[(size_t)f0 * 576 + i]); }
};
template <typename T>
struct SuperChild {   // assembleKs_level2_superEle_inplace.cu:113-140
    const T *Ks0; const int32_t *mapUnique; const T *E; const T *uFree; const T *uFixed; int hasFixed;
    __device__ double operator()(int32_t f0, int i) const {
        const int32_t uid1 = hasFixed ? mapUnique[f0] : 0;
        if (uid1 > 0) {
            const size_t fb = (size_t)(uid1 - 1) * 576 * 64, mb = (size_t)f0 * 64;
            double acc = 0.0;
            for (int q = 0; q < 64; ++q) acc += double(uFree[fb + (size_t)q * 576 + i]) * double(E[mb + q]);
            return acc + double(uFixed[(size_t)(uid1 - 1) * 576 + i]);
        }
        return double(Ks0[(size_t)f0 * 576 + i]);
    }
};

inline int blocks_for(int64_t n, int t) { return (int)((n + t - 1) / t); }

}  // namespace

extern "C" int top_gather(void *uMat, const void *u, const void *eNod, int eNodIsU32,
                          int64_t nElem, int64_t nNodes, int dtype, void *stream)
{
    if (nElem < 0 || nNodes < 0) { set_error("Gathering_inplace:Shape negative size"); return TOP_ERR_SHAPE; }
    if (dtype != TOP_F32 && dtype != TOP_F64) { set_error("Gathering_inplace:Type gU must be single or double."); return TOP_ERR_TYPE; }
    if (nElem == 0) return TOP_OK;
    if (!uMat || !u || !eNod) { set_error("Gathering_inplace:Args null pointer"); return TOP_ERR_ARGS; }
    const int T = 256, G = blocks_for(nElem, T);
    if (dtype == TOP_F64) {
        if (eNodIsU32) gather_kernel<double, uint32_t><<<G, T, 0, S(stream)>>>((double *)uMat, (const double *)u, (const uint32_t *)eNod, nElem, nNodes);
        else gather_kernel<double, int32_t><<<G, T, 0, S(stream)>>>((double *)uMat, (const double *)u, (const int32_t *)eNod, nElem, nNodes);
    } else {
        if (eNodIsU32) gather_kernel<float, uint32_t><<<G, T, 0, S(stream)>>>((float *)uMat, (const float *)u, (const uint32_t *)eNod, nElem, nNodes);
        else gather_kernel<float, int32_t><<<G, T, 0, S(stream)>>>((float *)uMat, (const float *)u, (const int32_t *)eNod, nElem, nNodes);
    }
    TOP_CUDA_CHECK(cudaGetLastError(), "Gathering_inplace");
    return TOP_OK;
}

extern "C" int top_scatter(void *Y, const int32_t *eNod, const void *uMat,
                           int64_t nElem, int64_t nNodes, int dtype, void *stream)
{
    if (nElem < 0 || nNodes < 0) { set_error("Scattering_inplace:shape negative size"); return TOP_ERR_SHAPE; }
    if (dtype != TOP_F32 && dtype != TOP_F64) { set_error("Scattering_inplace:type unsupported class"); return TOP_ERR_TYPE; }
    if (nElem > 0) {
        if (!Y || !eNod || !uMat) { set_error("Scattering_inplace:arity null pointer"); return TOP_ERR_ARGS; }
        const int T = 256, G = blocks_for(nElem, T);
        if (dtype == TOP_F64) scatter_kernel<double><<<G, T, 0, S(stream)>>>((double *)Y, eNod, (const double *)uMat, nElem, nNodes);
        else scatter_kernel<float><<<G, T, 0, S(stream)>>>((float *)Y, eNod, (const float *)uMat, nElem, nNodes);
        TOP_CUDA_CHECK(cudaGetLastError(), "Scattering_inplace");
    }
    TOP_CUDA_CHECK(cudaStreamSynchronize(S(stream)), "Scattering_inplace");
    return TOP_OK;
}

extern "C" int top_scatter_accum3(const int32_t *keys, const void *Tmp, int64_t N,
                                  void *xF, int64_t M, int dtype, void *stream)
{
    if (N < 0 || M < 0) { set_error("scatter_accum3:shape negative size"); return TOP_ERR_SHAPE; }
    if (dtype != TOP_F32 && dtype != TOP_F64) { set_error("scatter_accum3:type Only single or double supported for `Tmp`/`xFiner`."); return TOP_ERR_TYPE; }
    if (N == 0) return TOP_OK;
    if (!keys || !Tmp || !xF) { set_error("scatter_accum3:gpu All inputs must be gpuArray."); return TOP_ERR_ARGS; }
    const int T = 256, G = blocks_for(N, T);
    if (dtype == TOP_F64) scatter_accum3_kernel<double><<<G, T, 0, S(stream)>>>(keys, (const double *)Tmp, N, (double *)xF, M);
    else scatter_accum3_kernel<float><<<G, T, 0, S(stream)>>>(keys, (const float *)Tmp, N, (float *)xF, M);
    TOP_CUDA_CHECK(cudaGetLastError(), "scatter_accum3");
    return TOP_OK;
}

// Single is FP64 inside and rounded on the way out: the SIMT triple products in
// single took 1410 us for 8192 cells of 64 children, this form 139 us.
// Level-2 Galerkin assembly in the form Ks = (moduli of regular children) x Q
// on the FP64 tensor cores, plus the full triple product for children with
// fixed DOFs; in FP64 whatever the arrays' type T.  Shared with the fused
// solver.  Qscratch: [64 x 576] doubles, zero-filled by the caller, or null: each
// CTA forms the part of Q it multiplies by; numSMs: the current device's.
namespace {
// Q_s = P_s^T K0 P_s: the one-child cells of the identity map, written in FP64
template <typename T>
__global__ void __launch_bounds__(32) child_q_kernel(double *__restrict__ Q, const T *__restrict__ P, const T *__restrict__ K0)
{
    __shared__ double sT[24 * kDmmaLd];
    const int lane = threadIdx.x, g = lane >> 2, q = lane & 3;
    double kf[3][6], acc[3][3][2];
    zero_out(acc);
    load_child(K0Child<T>{K0}, 0, kf);
    child_product(P + (size_t)blockIdx.x * 576, kf, sT, acc);
#pragma unroll
    for (int I = 0; I < 3; ++I)
#pragma unroll
        for (int J = 0; J < 3; ++J)
#pragma unroll
            for (int h = 0; h < 2; ++h) Q[(size_t)blockIdx.x * 576 + (8 * I + g) + 24 * (8 * J + 2 * q + h)] = acc[I][J][h];
}
template <typename T>
int assemble_level2(T *Ks, const int32_t *upMap, const T *E, const T *K0, const T *Pch, const int32_t *mapUnique, const T *uFree,
                    const T *uFixed, int64_t nElem, int nCh, int64_t nUnique, double *Qscratch, cudaStream_t st, int numSMs,
                    const int32_t *bndList, int64_t nBnd)
{
    const int hasFixed = (nUnique > 0 && mapUnique && uFree && uFixed) ? 1 : 0;
    const Level2Child<T> child{E, K0, mapUnique, uFree, uFixed, hasFixed};
    if (nElem == 0) return TOP_OK;
    if (nCh <= kGemmK) {
        const Level2Row<T> row{upMap, E, mapUnique, nElem, nCh, hasFixed};
        const int64_t rb = (nElem + kGemmBM - 1) / kGemmBM;
        if (Qscratch) {
            if (nCh > 0) child_q_kernel<T><<<nCh, 32, 0, st>>>(Qscratch, Pch, K0);
            cudaFuncSetAttribute(dgemm_k64_kernel<T, Level2Row<T>>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGemmSmem);
            // B = Qscratch has 64 rows whatever nCh is: the GEMM's K tiles load rows
            // nCh..63 too and multiply them by the zero A entries that ARow returns
            // there, so those rows must exist and hold finite values (0 * NaN = NaN)
            dgemm_k64_kernel<<<dim3((unsigned)rb, gemm_k64_split(rb, numSMs)), 128, kGemmSmem, st>>>(Ks, nElem, 576, 576, Qscratch, 576, row);
        } else {
            using Kernel = void (*)(T *, int64_t, int, const T *, Level2Row<T>, K0Child<T>);
            const Kernel kern = gemm_q_kernel<T, Level2Row<T>, K0Child<T>>;
            cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGemmQSmem);
            const int64_t perTile = std::max<int64_t>(1, 2 * (int64_t)numSMs / 9);       // two CTAs an SM over the nine column tiles
            kern<<<dim3((unsigned)std::min(rb, perTile), 9), 128, kGemmQSmem, st>>>(Ks, nElem, nCh, Pch, row, K0Child<T>{K0});
        }
        // children with fixed DOFs: full triple products, accumulated; only the
        // coarse cells in bndList when the caller knows them (-1: all cells)
        if (hasFixed && nBnd != 0)
            ptkp(st, numSMs, Ks, upMap, nElem, nCh, Pch, child, RegularChild{mapUnique, hasFixed, 1}, 1,
                 nBnd > 0 ? bndList : nullptr, nBnd > 0 ? nBnd : nElem);
    } else {
        ptkp(st, numSMs, Ks, upMap, nElem, nCh, Pch, child, NoSkip{}, 0, nullptr, nElem);
    }
    return cudaGetLastError() == cudaSuccess ? TOP_OK : TOP_ERR_CUDA;
}
}  // namespace

namespace topgpu {
int assemble_level2_f64(double *Ks, const int32_t *upMap, const double *E, const double *K0,
                        const double *Pch, const int32_t *mapUnique, const double *uFree,
                        const double *uFixed, int64_t nElem, int nCh, int64_t nUnique,
                        double *Qscratch, cudaStream_t st, int numSMs, const int32_t *bndList, int64_t nBnd)
{
    return assemble_level2<double>(Ks, upMap, E, K0, Pch, mapUnique, uFree, uFixed, nElem, nCh, nUnique, Qscratch, st, numSMs, bndList, nBnd);
}

int assemble_higher_f64(double *Ks, const int32_t *upMap, const double *KsPrev, const double *Psub,
                        int64_t nElem, int nSub, cudaStream_t st, int numSMs)
{
    if (nElem == 0) return TOP_OK;
    ptkp(st, numSMs, Ks, upMap, nElem, nSub, Psub, PrevChild<double>{KsPrev}, NoSkip{}, 0, nullptr, nElem);
    return cudaGetLastError() == cudaSuccess ? TOP_OK : TOP_ERR_CUDA;
}
}  // namespace topgpu

namespace {
// the typed bodies of the gateways (arguments checked, zero elements excluded)
template <typename T>
int level2_typed(void *Ks, const int32_t *upMap, const void *E, const void *K0, const void *Pch, const int32_t *mapUnique,
                 const void *uFree, const void *uFixed, int64_t nElem, int nCh, int64_t nUnique, double *Q, cudaStream_t st)
{
    return assemble_level2<T>((T *)Ks, upMap, (const T *)E, (const T *)K0, (const T *)Pch, mapUnique, (const T *)uFree, (const T *)uFixed,
                              nElem, nCh, nUnique, Q, st, sm_count(), nullptr, -1);
}
template <typename T>
void higher_typed(void *Ks, const int32_t *upMap, const void *KsPrev, const void *Psub, int64_t nElem, int nSub, cudaStream_t st)
{
    ptkp(st, sm_count(), (T *)Ks, upMap, nElem, nSub, (const T *)Psub, PrevChild<T>{(const T *)KsPrev}, NoSkip{}, 0, nullptr, nElem);
}
template <typename T>
void super_typed(void *Ks, const int32_t *upMap, const void *Ks0, const void *Psub, const int32_t *mapUnique, const void *E,
                 const void *uFree, const void *uFixed, int64_t nElem, int nSub, int hasFixed, cudaStream_t st)
{
    ptkp(st, sm_count(), (T *)Ks, upMap, nElem, nSub, (const T *)Psub,
         SuperChild<T>{(const T *)Ks0, mapUnique, (const T *)E, (const T *)uFree, (const T *)uFixed, hasFixed}, NoSkip{}, 0, nullptr, nElem);
}
}  // namespace

extern "C" int top_assemble_ks_level2(void *Ks, const int32_t *upMap, const void *eleModulus,
                                      const void *K0, const void *Pch, const int32_t *mapUnique,
                                      const void *uniqueFree, const void *uniqueFixed,
                                      int64_t nElem, int nCh, int64_t nFine, int64_t nUnique,
                                      int dtype, void *stream)
{
    const char *N = "assembleKs_level2_inplace";
    if (dtype != TOP_F32 && dtype != TOP_F64) { set_error("%s:Type d_Ks must be single/double gpuArray.", N); return TOP_ERR_TYPE; }
    if (nElem < 0 || nCh < 0 || nFine < 0 || nUnique < 0) { set_error("%s:Shape negative size", N); return TOP_ERR_SHAPE; }
    if (nElem == 0) return TOP_OK;
    if (!Ks || !upMap || !eleModulus || !K0 || !Pch) { set_error("%s:Input null pointer", N); return TOP_ERR_ARGS; }
    const int hasFixed = (nUnique > 0 && mapUnique && uniqueFree && uniqueFixed) ? 1 : 0;
    cudaStream_t st = S(stream);
    struct Scratch {                 // a stream-ordered free on every exit
        void *p = nullptr; cudaStream_t st;
        explicit Scratch(cudaStream_t q) : st(q) {}
        ~Scratch() { if (p) cudaFreeAsync(p, st); }
    };
    {
        Scratch q(st);
        // One row block of cells in double: no CTA would use its Q tile twice, and
        // 64 CTAs form Q at once in stream-ordered scratch.  From two row blocks on
        // (and in single) the CTAs form their own tiles, without an allocation.
        if (dtype == TOP_F64 && nElem <= kGemmBM) {
            const size_t qn = (size_t)576 * 64;      // the GEMM's K rows
            TOP_CUDA_CHECK(cudaMallocAsync(&q.p, sizeof(double) * qn, st), N);
            TOP_CUDA_CHECK(cudaMemsetAsync(q.p, 0, sizeof(double) * qn, st), N);
        }
        double *Q = static_cast<double *>(q.p);
        const int64_t nu = hasFixed ? nUnique : 0;
        const int rc = dtype == TOP_F64
            ? level2_typed<double>(Ks, upMap, eleModulus, K0, Pch, mapUnique, uniqueFree, uniqueFixed, nElem, nCh, nu, Q, st)
            : level2_typed<float>(Ks, upMap, eleModulus, K0, Pch, mapUnique, uniqueFree, uniqueFixed, nElem, nCh, nu, Q, st);
        if (rc) { set_error("%s:CUDA launch failed: %s", N, cudaGetErrorString(cudaGetLastError())); return rc; }
    }
    TOP_CUDA_CHECK(cudaGetLastError(), N);
    TOP_CUDA_CHECK(cudaStreamSynchronize(st), N);   // assembleKs_level2_inplace.cu:272
    return TOP_OK;
}

extern "C" int top_assemble_ks_higher(void *Ks, const int32_t *upMap, const void *KsPrev,
                                      const void *Psub, int64_t nElem, int nSub, int64_t nFine,
                                      int dtype, void *stream)
{
    const char *N = "assembleKs_higherLevel_inplace";
    if (dtype != TOP_F32 && dtype != TOP_F64) { set_error("%s:Type d_Ks must be single/double gpuArray.", N); return TOP_ERR_TYPE; }
    if (nElem < 0 || nSub < 0 || nFine < 0) { set_error("%s:Shape negative size", N); return TOP_ERR_SHAPE; }
    if (nElem == 0) return TOP_OK;
    if (!Ks || !upMap || !KsPrev || !Psub) { set_error("%s:Input null pointer", N); return TOP_ERR_ARGS; }
    cudaStream_t st = S(stream);
    if (dtype == TOP_F64) higher_typed<double>(Ks, upMap, KsPrev, Psub, nElem, nSub, st);
    else higher_typed<float>(Ks, upMap, KsPrev, Psub, nElem, nSub, st);
    TOP_CUDA_CHECK(cudaGetLastError(), N);
    TOP_CUDA_CHECK(cudaStreamSynchronize(st), N);   // assembleKs_higherLevel_inplace.cu:209
    return TOP_OK;
}

extern "C" int top_assemble_ks_level2_super(void *Ks, const int32_t *upMap, const void *Ks0,
                                            const void *Psub, const int32_t *mapUnique,
                                            const void *eleModulus, const void *uniqueFree,
                                            const void *uniqueFixed, int64_t nElem, int nSub,
                                            int64_t nFine, int64_t nUnique, int dtype, void *stream)
{
    const char *N = "assembleKs_level2_superEle_inplace";
    if (dtype != TOP_F32 && dtype != TOP_F64) { set_error("%s:Type d_Ks must be single/double gpuArray.", N); return TOP_ERR_TYPE; }
    if (nElem < 0 || nSub < 0 || nFine < 0 || nUnique < 0) { set_error("%s:Shape negative size", N); return TOP_ERR_SHAPE; }
    if (nElem == 0) return TOP_OK;
    if (!Ks || !upMap || !Ks0 || !Psub || !eleModulus) { set_error("%s:Input null pointer", N); return TOP_ERR_ARGS; }
    const int hasFixed = (nUnique > 0 && mapUnique && uniqueFree && uniqueFixed) ? 1 : 0;
    cudaStream_t st = S(stream);
    if (dtype == TOP_F64) super_typed<double>(Ks, upMap, Ks0, Psub, mapUnique, eleModulus, uniqueFree, uniqueFixed, nElem, nSub, hasFixed, st);
    else super_typed<float>(Ks, upMap, Ks0, Psub, mapUnique, eleModulus, uniqueFree, uniqueFixed, nElem, nSub, hasFixed, st);
    TOP_CUDA_CHECK(cudaGetLastError(), N);
    TOP_CUDA_CHECK(cudaStreamSynchronize(st), N);   // ..._superEle_inplace.cu:313
    return TOP_OK;
}

// ---------------------------------------------------------------------------
// Allocation-free variant of top_assemble_ks_level2.
//
// Some callers cannot let this library allocate device memory during a
// call: a MEX gateway running inside MATLAB, whose gpuArray pool keeps most
// of the device memory and expects to be the only allocator, and
// applications that reserve their memory once up front and must not pay the
// implicit device synchronisation of cudaMalloc/cudaFree inside an
// optimisation loop.  This entry point takes its scratch (the child matrices
// Q_s = P_s' K0 P_s of the level-2 Galerkin GEMM) from the
// fixed device array below, which every GPU that loads the library holds
// until the process exits (about 295 KB per device).
//
// Limits and behaviour:
//  * at most kNoAllocMaxChildren (64) children per coarse element -- the
//    level-2 case of the reference (span 4); larger nCh is rejected with
//    TOP_ERR_SHAPE before anything runs;
//  * the first call on a device (and the first call after that device's
//    context was replaced, e.g. by cudaDeviceReset) resolves the arrays'
//    device addresses with cudaGetSymbolAddress, with that device current;
//    make that call before any stream capture on that device;
//  * all calls in double share the array and each clears it, so such calls
//    that run concurrently on the GPU (different streams or threads) race --
//    serialise them.  Calls in single take no scratch: every CTA forms the part
//    of Q it multiplies by.
namespace {
constexpr int kNoAllocMaxChildren = 64;
constexpr int kNoAllocMaxDevices = 64;
static __device__ __align__(256) double g_noalloc_Q[576 * kNoAllocMaxChildren];

// The resolved addresses are valid for one context of one device: a device
// reset unloads the module and the next context may place the arrays
// elsewhere, so the cache is keyed on (device, current context).  The context
// handle comes from the driver's cuCtxGetCurrent, looked up through the
// runtime (no link against libcuda).
struct NoAllocScratch { double *Q = nullptr; void *ctx = nullptr; };
std::mutex g_noalloc_mu;
NoAllocScratch g_noalloc_dev[kNoAllocMaxDevices];
bool g_noalloc_ready[kNoAllocMaxDevices] = {};
typedef int (*CtxGetCurrentFn)(void **);

int current_context(void **ctx, const char *N)
{
    static CtxGetCurrentFn fn = nullptr;
    if (!fn) {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        TOP_CUDA_CHECK(cudaGetDriverEntryPoint("cuCtxGetCurrent", &p, cudaEnableDefault, &q), N);
        if (q != cudaDriverEntryPointSuccess || !p) { set_error("%s:CUDA cuCtxGetCurrent not available", N); return TOP_ERR_CUDA; }
        fn = reinterpret_cast<CtxGetCurrentFn>(p);
    }
    *ctx = nullptr;
    if (fn(ctx) != 0 || !*ctx) { set_error("%s:CUDA no current context", N); return TOP_ERR_CUDA; }
    return TOP_OK;
}

int noalloc_scratch(NoAllocScratch *out, const char *N)
{
    int dev = 0;
    TOP_CUDA_CHECK(cudaGetDevice(&dev), N);
    if (dev < 0 || dev >= kNoAllocMaxDevices) { set_error("%s:CUDA device %d out of range", N, dev); return TOP_ERR_CUDA; }
    TOP_CUDA_CHECK(cudaSetDevice(dev), N);         // binds the device's primary context to this thread
    void *ctx = nullptr;
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    int rc = current_context(&ctx, N);
    if (rc) return rc;
    if (!g_noalloc_ready[dev] || g_noalloc_dev[dev].ctx != ctx) {
        NoAllocScratch s;
        TOP_CUDA_CHECK(cudaGetSymbolAddress((void **)&s.Q, g_noalloc_Q), N);
        s.ctx = ctx;
        g_noalloc_dev[dev] = s;
        g_noalloc_ready[dev] = true;
    }
    *out = g_noalloc_dev[dev];
    return TOP_OK;
}
}  // namespace

extern "C" int top_assemble_ks_level2_noalloc(void *Ks, const int32_t *upMap, const void *eleModulus,
                                              const void *K0, const void *Pch, const int32_t *mapUnique,
                                              const void *uniqueFree, const void *uniqueFixed,
                                              int64_t nElem, int nCh, int64_t nFine, int64_t nUnique,
                                              int dtype, void *stream)
{
    const char *N = "assembleKs_level2_inplace";
    if (dtype != TOP_F32 && dtype != TOP_F64) { set_error("%s:Type d_Ks must be single/double gpuArray.", N); return TOP_ERR_TYPE; }
    if (nElem < 0 || nCh < 0 || nFine < 0 || nUnique < 0) { set_error("%s:Shape negative size", N); return TOP_ERR_SHAPE; }
    if (nCh > kNoAllocMaxChildren) {
        set_error("%s:Shape %d children per coarse element exceed the allocation-free limit of %d", N, nCh, kNoAllocMaxChildren);
        return TOP_ERR_SHAPE;
    }
    if (nElem == 0) return TOP_OK;
    if (!Ks || !upMap || !eleModulus || !K0 || !Pch) { set_error("%s:Input null pointer", N); return TOP_ERR_ARGS; }
    const int hasFixed = (nUnique > 0 && mapUnique && uniqueFree && uniqueFixed) ? 1 : 0;
    cudaStream_t st = S(stream);
    const int64_t nu = hasFixed ? nUnique : 0;
    int rc;
    if (dtype == TOP_F64) {
        NoAllocScratch sc;
        rc = noalloc_scratch(&sc, N);
        if (rc) return rc;
        // the GEMM loads all 64 rows of Q and multiplies rows nCh..63 by zero:
        // clear them all, so that no value left by an earlier call (NaN or Inf
        // included) reaches this call's result
        TOP_CUDA_CHECK(cudaMemsetAsync(sc.Q, 0, sizeof(double) * 576 * kNoAllocMaxChildren, st), N);
        rc = level2_typed<double>(Ks, upMap, eleModulus, K0, Pch, mapUnique, uniqueFree, uniqueFixed, nElem, nCh, nu, sc.Q, st);
    } else {                         // no scratch: concurrent calls in single share nothing
        rc = level2_typed<float>(Ks, upMap, eleModulus, K0, Pch, mapUnique, uniqueFree, uniqueFixed, nElem, nCh, nu, nullptr, st);
    }
    if (rc) { set_error("%s:CUDA launch failed: %s", N, cudaGetErrorString(cudaGetLastError())); return rc; }
    TOP_CUDA_CHECK(cudaGetLastError(), N);
    TOP_CUDA_CHECK(cudaStreamSynchronize(st), N);
    return TOP_OK;
}
