// topgpu_kernels.cuh -- device kernels shared by the MEX drop-ins and the
// fused solver: Galerkin triple products and the FP64 tensor-core GEMM.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include "topgpu_internal.h"

#define TOP_CUDA_CHECK(call, name)                                                   \
    do {                                                                             \
        cudaError_t err__ = (call);                                                  \
        if (err__ != cudaSuccess) {                                                  \
            topgpu::set_error("%s:CUDA CUDA error %d: %s", name, (int)err__,         \
                              cudaGetErrorString(err__));                            \
            return TOP_ERR_CUDA;                                                     \
        }                                                                            \
    } while (0)

namespace topgpu {

// ---------------------------------------------------------------------------
// FP64 tensor-core GEMM  C[M x N] (row-major, ldc) = A[M x 64] * B[64 x N]
// with mma.sync.m8n8k4.f64 (the FP64 tensor path of sm_100a), C rounded to its
// storage type.  A's rows are produced on the fly by ARow (e.g. child moduli of
// a coarse cell); B is row-major [64 x ldb].  CTA tile 64 x 64, 4 warps of
// 32 x 32; gridDim.y CTAs share a row block's column tiles.
constexpr int kGemmBM = 64, kGemmBN = 64, kGemmK = 64, kGemmPad = 4;

__device__ __forceinline__ void dmma_8x8x4(double &d0, double &d1, double a, double b)
{
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
                 : "+d"(d0), "+d"(d1) : "d"(a), "d"(b));
}

// one 64 x 64 tile of C from the staged A [64][K + pad] and B [K][64 + pad]
template <typename T>
__device__ __forceinline__ void gemm_k64_tile(T *__restrict__ C, int64_t M, int N, int64_t ldc, int64_t m0, int n0,
                                              const double *sA, const double *sB)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int wr = (warp & 1) * 32, wc = (warp >> 1) * 32;
    const int g = lane >> 2, q = lane & 3;
    double acc[4][4][2];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
#pragma unroll 4
    for (int k0 = 0; k0 < kGemmK; k0 += 4) {
        double a[4], b[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) a[i] = sA[(wr + 8 * i + g) * (kGemmK + kGemmPad) + k0 + q];
#pragma unroll
        for (int j = 0; j < 4; ++j) b[j] = sB[(k0 + q) * (kGemmBN + kGemmPad) + wc + 8 * j + g];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) dmma_8x8x4(acc[i][j][0], acc[i][j][1], a[i], b[j]);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int64_t m = m0 + wr + 8 * i + g;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + wc + 8 * j + 2 * q;
            if (n < N) C[m * ldc + n] = T(acc[i][j][0]);
            if (n + 1 < N) C[m * ldc + n + 1] = T(acc[i][j][1]);
        }
    }
}

// the A tile of rows m0 .. m0 + 63: arow.child(m, k) (the child's 1-based id, 0:
// none) for eight pairs a thread, then their arow.value's, so that each of the
// dependent loads is issued eight times before the next waits (one pair after
// another a tile's gather took 34 us)
template <class ARow>
__device__ __forceinline__ void gather_a(double *sA, const ARow &arow, int64_t m0, int64_t M)
{
    for (int u0 = 0; u0 < kGemmBM * kGemmK / 128; u0 += 8) {
        int32_t f[8];
        double v[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int idx = threadIdx.x + 128 * (u0 + u), r = idx % kGemmBM, k = idx / kGemmBM;
            f[u] = m0 + r < M ? arow.child(m0 + r, k) : 0;
        }
#pragma unroll
        for (int u = 0; u < 8; ++u) v[u] = f[u] > 0 ? arow.value(f[u] - 1) : 0.0;
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            const int idx = threadIdx.x + 128 * (u0 + u), r = idx % kGemmBM, k = idx / kGemmBM;
            sA[r * (kGemmK + kGemmPad) + k] = f[u] > 0 && arow.regular(f[u] - 1) ? v[u] : 0.0;
        }
    }
}

template <typename T, class ARow>
__global__ void __launch_bounds__(128)
dgemm_k64_kernel(T *__restrict__ C, int64_t M, int N, int64_t ldc,
                 const double *__restrict__ B, int ldb, ARow arow)
{
    extern __shared__ double smem[];
    double *sA = smem;                                  // [BM][K + pad]
    double *sB = smem + kGemmBM * (kGemmK + kGemmPad);  // [K][BN + pad]
    const int64_t m0 = (int64_t)blockIdx.x * kGemmBM;
    const int tid = threadIdx.x;
    // A tile once per CTA
    gather_a(sA, arow, m0, M);
    // the CTA's column tiles in turn, the A tile reused from shared memory
    for (int n0 = blockIdx.y * kGemmBN; n0 < N; n0 += gridDim.y * kGemmBN) {
        __syncthreads();                                    // sB free (and sA complete)
#pragma unroll 8
        for (int u = 0; u < kGemmK * kGemmBN / 128; ++u) {
            const int idx = tid + 128 * u, k = idx / kGemmBN, c = idx % kGemmBN;
            sB[k * (kGemmBN + kGemmPad) + c] = (n0 + c < N) ? B[(size_t)k * ldb + n0 + c] : 0.0;
        }
        __syncthreads();
        gemm_k64_tile(C, M, N, ldc, m0, n0, sA, sB);
    }
}

constexpr size_t kGemmSmem = sizeof(double) * (kGemmBM * (kGemmK + kGemmPad) + kGemmK * (kGemmBN + kGemmPad));

// CTAs that share a row block's nine column tiles of 64 (576 outputs): enough for
// two CTAs an SM where the row blocks alone are fewer.  Each CTA gathers the A
// tile for itself, so one CTA a row block is best once they fill the chip (432
// row blocks: assembly 1.50 -> 1.37 ms).  With one CTA a row block 7 row blocks
// took 106 us and 128 took 104; nine and three CTAs, with the gathers batched,
// bring the whole assembly of 24x48x24 from 318 to 230 us and of 64x128x64 from
// 924 to 839.
inline unsigned gemm_k64_split(int64_t rowBlocks, int numSMs)
{
    for (unsigned y : {1u, 3u})
        if (rowBlocks * y >= 2 * (int64_t)numSMs) return y;
    return 9;
}

// ---------------------------------------------------------------------------
// Galerkin triple products on the FP64 tensor cores: Kout = sum over children
// of P_s^T (K_s P_s), every 24 x 24 product as 3 x 3 tiles of
// mma.sync.m8n8k4.f64 (six k-steps each: 108 MMAs per child), in FP64 whatever
// the matrices' storage type T.  A lane reads the fragments of K_s and P_s it
// needs straight from global memory (columns' 64-byte pieces; P_s, one small
// matrix a child slot shared by every warp, from L1); only T = K_s P_s changes
// layout through shared memory (leading dimension 25).  childK(f0, i) yields
// entry i (column-major) of child f0's matrix, the child list is upMap[e + s
// nElem] (1-based, <= 0 = skip) and skip(f0) excludes children handled
// elsewhere.  The chain upMap -> K_s -> MMAs of one child bounds a warp, so
// the next child's index and matrix are loaded during this one's MMAs.
constexpr int kDmmaWarps = 4;
constexpr int kDmmaLd = 25;

// next child at or after s (stride step) that is not skipped; nCh when none
template <class Skip>
__device__ __forceinline__ int next_child(const int32_t *upMap, int64_t e, int64_t nElem, int nCh, int s, int step, const Skip &skip, int32_t &f0)
{
    for (; s < nCh; s += step) {
        const int32_t f1 = upMap[e + (int64_t)s * nElem];
        if (f1 > 0 && !skip(f1 - 1)) { f0 = f1 - 1; return s; }
    }
    return nCh;
}
template <class ChildK>
__device__ __forceinline__ void load_child(const ChildK &childK, int32_t f0, double (&kf)[3][6])
{
    const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
#pragma unroll
    for (int kk = 0; kk < 6; ++kk)
#pragma unroll
        for (int I = 0; I < 3; ++I) kf[I][kk] = double(childK(f0, (8 * I + g) + 24 * (4 * kk + q)));
}
// acc += P_s^T (K_s P_s) with K_s in fragments; sT: the warp's 24 x 25 scratch
template <typename T>
__device__ __forceinline__ void child_product(const T *__restrict__ Ps, const double (&kf)[3][6], double *sT, double (&acc)[3][3][2])
{
    const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
    // T = K_s P_s: tile (I, J) = sum_kk K[8I.., 4kk..] P[4kk.., 8J..]
#pragma unroll
    for (int J = 0; J < 3; ++J) {
        double b[6];
#pragma unroll
        for (int kk = 0; kk < 6; ++kk) b[kk] = double(__ldg(Ps + (4 * kk + q) + 24 * (8 * J + g)));
        double d[3][2];
#pragma unroll
        for (int I = 0; I < 3; ++I) d[I][0] = d[I][1] = 0.0;
#pragma unroll
        for (int kk = 0; kk < 6; ++kk)
#pragma unroll
            for (int I = 0; I < 3; ++I) dmma_8x8x4(d[I][0], d[I][1], kf[I][kk], b[kk]);
#pragma unroll
        for (int I = 0; I < 3; ++I) {
            sT[(8 * I + g) + kDmmaLd * (8 * J + 2 * q)] = d[I][0];
            sT[(8 * I + g) + kDmmaLd * (8 * J + 2 * q + 1)] = d[I][1];
        }
    }
    __syncwarp();
    // Kout += P_s^T T: A = P^T (8I.., 4kk..) = P(4kk.., 8I..), B = T(4kk.., 8J..)
#pragma unroll
    for (int I = 0; I < 3; ++I) {
        double a[6];
#pragma unroll
        for (int kk = 0; kk < 6; ++kk) a[kk] = double(__ldg(Ps + (4 * kk + q) + 24 * (8 * I + g)));
#pragma unroll
        for (int kk = 0; kk < 6; ++kk)
#pragma unroll
            for (int J = 0; J < 3; ++J) dmma_8x8x4(acc[I][J][0], acc[I][J][1], a[kk], sT[(4 * kk + q) + kDmmaLd * (8 * J + g)]);
    }
    __syncwarp();                                    // sT is rewritten by the next child
}
__device__ __forceinline__ void zero_out(double (&acc)[3][3][2])
{
#pragma unroll
    for (int I = 0; I < 3; ++I)
#pragma unroll
        for (int J = 0; J < 3; ++J) acc[I][J][0] = acc[I][J][1] = 0.0;
}

// one coarse element per warp
template <typename T, class ChildK, class Skip>
__global__ void __launch_bounds__(32 * kDmmaWarps)
ptkp_dmma_kernel(T *__restrict__ Ks, const int32_t *__restrict__ upMap, int64_t nElem, int nCh,
                 const T *__restrict__ P, ChildK childK, Skip skip, int accumulate,
                 const int32_t *__restrict__ elist, int64_t nSel)
{
    __shared__ double smem[kDmmaWarps][24 * kDmmaLd];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
    const int64_t w = (int64_t)blockIdx.x * kDmmaWarps + warp;
    if (w >= nSel) return;                           // whole warps; no CTA-wide barrier below
    const int64_t e = elist ? (int64_t)elist[w] : w;
    double acc[3][3][2], kf[3][6];
    zero_out(acc);
    int32_t f0 = 0;
    int s = next_child(upMap, e, nElem, nCh, 0, 1, skip, f0);
    const bool any = s < nCh;
    if (any) load_child(childK, f0, kf);
    while (s < nCh) {
        double kn[3][6];
        const int sn = next_child(upMap, e, nElem, nCh, s + 1, 1, skip, f0);
        if (sn < nCh) load_child(childK, f0, kn);
        child_product(P + (size_t)s * 576, kf, smem[warp], acc);
#pragma unroll
        for (int I = 0; I < 3; ++I)
#pragma unroll
            for (int kk = 0; kk < 6; ++kk) kf[I][kk] = kn[I][kk];
        s = sn;
    }
    if (accumulate && !any) return;
    T *out = Ks + (size_t)e * 576;
#pragma unroll
    for (int I = 0; I < 3; ++I)
#pragma unroll
        for (int J = 0; J < 3; ++J)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int idx = (8 * I + g) + 24 * (8 * J + 2 * q + h);
                out[idx] = T(accumulate ? double(out[idx]) + acc[I][J][h] : acc[I][J][h]);
            }
}
// Many children per coarse element (the 64 of a span-4 cell): a CTA's
// kSplitWarps warps take children w, w + kSplitWarps, ... of one element and the
// warps' partial sums are added in warp order through shared memory
// (deterministic), so a level with few coarse elements still fills the GPU.
// probe (accumulating over every element, few of which have a child that is not
// skipped): the CTA first looks at all children of kProbe elements at once and
// forms only those that have one; element by element, each warp walking its
// skipped children in turn, took 215 us for 8192 elements with 256 of them.
constexpr int kSplitWarps = 8, kProbe = 4;

template <typename T, class ChildK, class Skip>
__global__ void __launch_bounds__(32 * kSplitWarps, 2)
ptkp_dmma_split_kernel(T *__restrict__ Ks, const int32_t *__restrict__ upMap, int64_t nElem, int nCh,
                       const T *__restrict__ P, ChildK childK, Skip skip, int accumulate,
                       const int32_t *__restrict__ elist, int64_t nSel, int probe)
{
    __shared__ double smem[kSplitWarps][24 * kDmmaLd];
    __shared__ int flag[kProbe + kSplitWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
    double *sT = smem[warp];
    int *anyW = flag + kProbe;
    const int group = probe ? kProbe : 1;
    for (int64_t i0 = blockIdx.x; i0 < nSel; i0 += (int64_t)gridDim.x * group) {
        if (probe) {
            __syncthreads();                         // the previous group's flags are read
            if (threadIdx.x < kProbe) flag[threadIdx.x] = 0;
            __syncthreads();
            constexpr int per = 32 * kSplitWarps / kProbe;
            const int j = threadIdx.x / per;
            const int64_t w = i0 + (int64_t)j * gridDim.x;
            if (w < nSel)
                for (int c = threadIdx.x % per; c < nCh; c += per) {
                    const int32_t f1 = upMap[w + (int64_t)c * nElem];
                    if (f1 > 0 && !skip(f1 - 1)) flag[j] = 1;
                }
            __syncthreads();
        }
        for (int j = 0; j < group; ++j) {
            const int64_t w = i0 + (int64_t)j * gridDim.x;
            if (w >= nSel || (probe && !flag[j])) continue;          // uniform in the CTA
            const int64_t e = elist ? (int64_t)elist[w] : w;
            double acc[3][3][2];
            zero_out(acc);
            int32_t f0 = 0;
            bool any = false;
            for (int s = next_child(upMap, e, nElem, nCh, warp, kSplitWarps, skip, f0); s < nCh;
                 s = next_child(upMap, e, nElem, nCh, s + kSplitWarps, kSplitWarps, skip, f0)) {
                double kf[3][6];
                load_child(childK, f0, kf);
                child_product(P + (size_t)s * 576, kf, sT, acc);
                any = true;
            }
            // the warp's scratch now takes its partial sums
#pragma unroll
            for (int I = 0; I < 3; ++I)
#pragma unroll
                for (int J = 0; J < 3; ++J)
#pragma unroll
                    for (int h = 0; h < 2; ++h) sT[(8 * I + g) + 24 * (8 * J + 2 * q + h)] = acc[I][J][h];
            if (lane == 0) anyW[warp] = any ? 1 : 0;
            __syncthreads();
            bool anyC = false;
            for (int v = 0; v < kSplitWarps; ++v) anyC = anyC || anyW[v];
            if (!(accumulate && !anyC)) {
                T *out = Ks + (size_t)e * 576;
                for (int i = threadIdx.x; i < 576; i += 32 * kSplitWarps) {
                    double v = smem[0][i];
#pragma unroll
                    for (int u = 1; u < kSplitWarps; ++u) v += smem[u][i];
                    out[i] = T(accumulate ? double(out[i]) + v : v);
                }
            }
            __syncthreads();                         // the scratch is reused
        }
    }
}

// launch over nSel coarse elements (elist, or 0 .. nSel-1): children split
// over the warps of a CTA when a cell has many, one warp per cell otherwise;
// an accumulating launch over all cells probes them first
template <typename T, class ChildK, class Skip>
inline void ptkp(cudaStream_t st, int numSMs, T *Ks, const int32_t *upMap, int64_t nElem, int nCh, const T *P,
                 ChildK childK, Skip skip, int accumulate, const int32_t *elist, int64_t nSel)
{
    if (nSel <= 0) return;
    if (nCh >= 2 * kSplitWarps) {
        const int probe = accumulate && !elist ? 1 : 0;
        const unsigned grid = probe ? (unsigned)((nSel + kProbe - 1) / kProbe < 2 * (int64_t)numSMs ? (nSel + kProbe - 1) / kProbe : 2 * (int64_t)numSMs)
                                    : (unsigned)nSel;
        ptkp_dmma_split_kernel<T, ChildK, Skip><<<grid, 32 * kSplitWarps, 0, st>>>(Ks, upMap, nElem, nCh, P, childK, skip, accumulate,
                                                                                 elist, nSel, probe);
        return;
    }
    ptkp_dmma_kernel<T, ChildK, Skip><<<(unsigned)((nSel + kDmmaWarps - 1) / kDmmaWarps), 32 * kDmmaWarps, 0, st>>>(
        Ks, upMap, nElem, nCh, P, childK, skip, accumulate, elist, nSel);
}
// The same GEMM with B formed by the CTA itself: column tile blockIdx.y (64 of
// the 576 entries) of Q_s = P_s^T K0 P_s for the nCh <= 64 children, each warp 16
// of them (the same MMAs as a whole triple product's, for the one or two
// 8-column groups the tile touches), then the row blocks blockIdx.x, blockIdx.x +
// gridDim.x, ... with it.  Needs no scratch in global memory: a stream-ordered
// allocation of it cost about 400 us a call where the pool hands its memory back
// at every synchronisation (8192 cells: 567 -> 147 us a call without it).
constexpr size_t kGemmQSmem = kGemmSmem + sizeof(double) * kDmmaWarps * 24 * kDmmaLd;
template <typename T, class ARow, class ChildK>
__global__ void __launch_bounds__(32 * kDmmaWarps)
gemm_q_kernel(T *__restrict__ C, int64_t M, int nCh, const T *__restrict__ P, ARow arow, ChildK childK)
{
    extern __shared__ double smem[];
    constexpr int LB = kGemmBN + kGemmPad;
    double *sA = smem, *sB = smem + kGemmBM * (kGemmK + kGemmPad);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3;
    double *sT = sB + kGemmK * LB + warp * 24 * kDmmaLd;
    const int n0 = blockIdx.y * kGemmBN;
    {
        double kf[3][6], pn[3][6];
        load_child(childK, 0, kf);
        // P_s fragments (4kk + q, 8I + g), the next child's loaded during this one's MMAs
        auto load_p = [&](int s, double (&p)[3][6]) {
#pragma unroll
            for (int I = 0; I < 3; ++I)
#pragma unroll
                for (int kk = 0; kk < 6; ++kk) p[I][kk] = double(__ldg(P + (size_t)s * 576 + (4 * kk + q) + 24 * (8 * I + g)));
        };
        if (warp < nCh) load_p(warp, pn);
        for (int s = warp; s < kGemmK; s += kDmmaWarps) {
            if (s >= nCh) {
                for (int c = lane; c < kGemmBN; c += 32) sB[s * LB + c] = 0.0;
                continue;
            }
            double p[3][6];
#pragma unroll
            for (int I = 0; I < 3; ++I)
#pragma unroll
                for (int kk = 0; kk < 6; ++kk) p[I][kk] = pn[I][kk];
            if (s + kDmmaWarps < nCh) load_p(s + kDmmaWarps, pn);
#pragma unroll
            for (int J = 0; J < 3; ++J) {                                        // 8 columns of 24 entries
                if (192 * J + 192 <= n0 || 192 * J >= n0 + kGemmBN) continue;      // uniform in the CTA
                double d[3][2];
#pragma unroll
                for (int I = 0; I < 3; ++I) d[I][0] = d[I][1] = 0.0;
#pragma unroll
                for (int kk = 0; kk < 6; ++kk)
#pragma unroll
                    for (int I = 0; I < 3; ++I) dmma_8x8x4(d[I][0], d[I][1], kf[I][kk], p[J][kk]);
                __syncwarp();
#pragma unroll
                for (int I = 0; I < 3; ++I) {
                    sT[(8 * I + g) + kDmmaLd * (2 * q)] = d[I][0];
                    sT[(8 * I + g) + kDmmaLd * (2 * q + 1)] = d[I][1];
                }
                __syncwarp();
                double o[3][2];
#pragma unroll
                for (int I = 0; I < 3; ++I) o[I][0] = o[I][1] = 0.0;
#pragma unroll
                for (int kk = 0; kk < 6; ++kk) {
                    const double t = sT[(4 * kk + q) + kDmmaLd * g];
#pragma unroll
                    for (int I = 0; I < 3; ++I) dmma_8x8x4(o[I][0], o[I][1], p[I][kk], t);
                }
#pragma unroll
                for (int I = 0; I < 3; ++I) {
                    const int n = (8 * I + g) + 24 * (8 * J + 2 * q) - n0;
                    if (n >= 0 && n < kGemmBN) sB[s * LB + n] = o[I][0];
                    if (n + 24 >= 0 && n + 24 < kGemmBN) sB[s * LB + n + 24] = o[I][1];
                }
            }
        }
    }
    for (int64_t rb = blockIdx.x; rb * kGemmBM < M; rb += gridDim.x) {
        __syncthreads();                             // sA free (and sB complete)
        const int64_t m0 = rb * kGemmBM;
        gather_a(sA, arow, m0, M);
        __syncthreads();
        gemm_k64_tile(C, M, 576, 576, m0, n0, sA, sB);
    }
}
inline int sm_count()
{
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    return n;
}

}  // namespace topgpu
