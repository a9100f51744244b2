// topgpu_dense.cuh -- dense FP64 linear algebra of the coarsest level: the
// Cholesky factor of the assembled coarsest matrix and its explicit inverse
// (the V-cycle's coarsest solve is one GEMV with it).
//
//   * factorisation: right-looking over 32-column blocks, taken 128 columns at
//     a time: chol_diag_kernel factors the 128 x 128 diagonal block in one
//     CTA's shared memory (and inverts its four 32 x 32 diagonal blocks),
//     chol_panel_kernel forms the panel below it, L21 = A21 L11^-T block by
//     block, and chol_trail_kernel applies the four rank-32 updates
//     A22 -= L21 L21^T to every trailing tile in one pass.  Each entry still
//     receives the 32-column blocks' contributions one after another, each
//     summed from zero, as a sweep of one block at a time gives them;
//   * W = L^-1 by 2x2 block inversion, [L11 0; L21 L22]^-1 =
//     [W11 0; -W22 L21 W11  W22], bottom-up from the factorisation's
//     diagonal blocks, every node of a level in one launch;
//   * A^-1 = W^T W on the lower tiles, mirrored, skipping the zero blocks of W.
//
// Measured on one B200, factor and inverse (bit-identical to the sweep of one
// 32-column block a step on SIMT tiles that this replaces): n = 336 506 -> 312
// us, n = 1386 2.31 -> 1.23 ms, n = 4131 12.4 -> 5.8 ms (the last factor and
// trailing updates 3.4 ms, W 1.4 ms, W^T W 0.9 ms; its 35 G multiply-adds take
// 2.5 ms at the FP64 peak).  Small sizes are bound by the diagonal blocks' chain
// of square roots and divisions, about 11 us a block of 32 columns.
//
// All products run on mma.sync.m8n8k4.f64 through one tile loop (64 x 64
// outputs, 4 warps of 32 x 32, K steps of 16 double-buffered in shared memory)
// over column-major matrices.  The FP64 tensor instruction adds its four
// products as a chain of fused multiply-adds in k order (compared bit for bit
// against that chain on the B200), and its rate there is the FP64 pipe's (18.5
// against 18.0 T multiply-adds/s), so it gives the sums of a plain multiply-add
// loop; what it saves is operand traffic: 8 shared-memory reads a lane feed 16
// instructions of 256 multiply-adds, against 16 multiply-adds a lane before.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include "topgpu_kernels.cuh"

namespace topgpu {

constexpr int kDb = 32;          // diagonal block of the factorisation
constexpr int kPb = 128;         // columns of one factorisation step (four blocks)

// ---- the tile loop ------------------------------------------------------------
// Shared-memory stage of a 64 x 16 operand piece: rows consecutive in memory
// (T false) at [k][68], k consecutive (T true) at [row][20]; both strides are 4
// modulo 16, so the (row 8, k 4) fragment of a half-warp covers the 16 banks pairs.
constexpr int kTileB = 64, kTileK = 16, kTileThreads = 128;
template <bool T> struct TileStage {
    static constexpr int vals = T ? kTileB * 20 : kTileK * 68;
    __device__ static int at(int row, int k) { return T ? row * 20 + k : k * 68 + row; }
    __device__ static void place(int e, int &row, int &k) { if (T) { k = e % kTileK; row = e / kTileK; } else { row = e % kTileB; k = e / kTileB; } }
};
template <bool TA, bool TB> constexpr int tile_smem_vals = 2 * (TileStage<TA>::vals + TileStage<TB>::vals);

// acc += sum over k in [kBeg, kEnd) of fa(row, k) fb(col, k) for the warp's
// 32 x 32 part (rows 32 (warp & 1) + 8 I + lane / 4, columns 32 (warp >> 1) + 8 J +
// 2 (lane % 4) + {0, 1}); fold() runs after every 32 values of k and at the end.
// fa / fb return 0 outside the matrices.
template <bool TA, bool TB, class FA, class FB, class Fold>
__device__ __forceinline__ void dmma_tile(FA fa, FB fb, int kBeg, int kEnd, double (&acc)[4][4][2], double *sm, Fold fold)
{
    constexpr int SA = TileStage<TA>::vals, SB = TileStage<TB>::vals;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5, g = lane >> 2, q = lane & 3;
    const int wr = (warp & 1) * 32, wc = (warp >> 1) * 32;
    double ra[8], rb[8];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            int row, k;
            TileStage<TA>::place(t + kTileThreads * u, row, k);
            ra[u] = k0 + k < kEnd ? fa(row, k0 + k) : 0.0;
            TileStage<TB>::place(t + kTileThreads * u, row, k);
            rb[u] = k0 + k < kEnd ? fb(row, k0 + k) : 0.0;
        }
    };
    if (kBeg < kEnd) fetch(kBeg);
    int buf = 0;
    for (int k0 = kBeg; k0 < kEnd; k0 += kTileK, buf ^= 1) {
        double *sa = sm + buf * (SA + SB), *sb = sa + SA;
#pragma unroll
        for (int u = 0; u < 8; ++u) {
            int row, k;
            TileStage<TA>::place(t + kTileThreads * u, row, k);
            sa[TileStage<TA>::at(row, k)] = ra[u];
            TileStage<TB>::place(t + kTileThreads * u, row, k);
            sb[TileStage<TB>::at(row, k)] = rb[u];
        }
        __syncthreads();                 // one barrier a step: the other buffer's readers are past it
        if (k0 + kTileK < kEnd) fetch(k0 + kTileK);
#pragma unroll
        for (int kk = 0; kk < kTileK; kk += 4) {
            double a[4], b[4];
#pragma unroll
            for (int I = 0; I < 4; ++I) a[I] = sa[TileStage<TA>::at(wr + 8 * I + g, kk + q)];
#pragma unroll
            for (int J = 0; J < 4; ++J) b[J] = sb[TileStage<TB>::at(wc + 8 * J + g, kk + q)];
#pragma unroll
            for (int I = 0; I < 4; ++I)
#pragma unroll
                for (int J = 0; J < 4; ++J) dmma_8x8x4(acc[I][J][0], acc[I][J][1], a[I], b[J]);
        }
        if (((k0 - kBeg) & kTileK) || k0 + kTileK >= kEnd) fold();
    }
}
struct NoFold { __device__ void operator()() const {} };
__device__ __forceinline__ void zero_acc(double (&acc)[4][4][2])
{
#pragma unroll
    for (int I = 0; I < 4; ++I)
#pragma unroll
        for (int J = 0; J < 4; ++J) acc[I][J][0] = acc[I][J][1] = 0.0;
}
// f(row, col, value) over the thread's outputs of a tile
template <class F>
__device__ __forceinline__ void each_out(double (&acc)[4][4][2], F f)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, q = lane & 3;
#pragma unroll
    for (int I = 0; I < 4; ++I)
#pragma unroll
        for (int J = 0; J < 4; ++J)
#pragma unroll
            for (int h = 0; h < 2; ++h) f((warp & 1) * 32 + 8 * I + g, (warp >> 1) * 32 + 8 * J + 2 * q + h, acc[I][J][h]);
}

// C(i, j) = sum_k a(i, k) b(j, k) for i < M, j < N, a(i, k) = TA ? A[k + lda i]
// : A[i + lda k] (likewise b).  lower: only tiles on or below the diagonal;
// mirror: those, and their transposes written above it (a symmetric product).
// kFromTile: a(i, k) = 0 and b(j, k) = 0 for k below the tile's first row /
// column (triangular factors), so K starts at max(i0, j0).
template <bool TA, bool TB>
__global__ void __launch_bounds__(kTileThreads)
dgemm_tile_kernel(double *C, int64_t ldc, const double *A, int64_t lda, const double *B, int64_t ldb,
                  int M, int N, int K, int lower, int mirror, int kFromTile)
{
    __shared__ double sm[tile_smem_vals<TA, TB>];
    const int i0 = blockIdx.x * kTileB, j0 = blockIdx.y * kTileB;
    if ((lower || mirror) && j0 > i0) return;
    double acc[4][4][2];
    zero_acc(acc);
    const int kStart = kFromTile ? ((i0 > j0 ? i0 : j0) / kTileK) * kTileK : 0;
    dmma_tile<TA, TB>([&](int r, int k) { const int i = i0 + r; return i < M ? (TA ? A[k + lda * i] : A[i + lda * k]) : 0.0; },
                      [&](int r, int k) { const int j = j0 + r; return j < N ? (TB ? B[k + ldb * j] : B[j + ldb * k]) : 0.0; },
                      kStart, K, acc, sm, NoFold{});
    each_out(acc, [&](int r, int c, double v) {
        const int i = i0 + r, j = j0 + c;
        if (i >= M || j >= N) return;
        C[i + ldc * j] = v;
        if (mirror && i0 != j0) C[j + ldc * i] = v;
    });
}

// A^-1 = W^T W as packed lower tiles: tile (I, J), J <= I, at index I (I + 1) / 2 + J,
// 64 x 64 column-major, zero past row or column n (the diagonal tiles whole)
__global__ void __launch_bounds__(kTileThreads)
wtw_packed_kernel(double *__restrict__ P, const double *__restrict__ W, int64_t n)
{
    __shared__ double sm[tile_smem_vals<true, true>];
    const int i0 = blockIdx.x * kTileB, j0 = blockIdx.y * kTileB;
    if (j0 > i0) return;
    double acc[4][4][2];
    zero_acc(acc);
    dmma_tile<true, true>([&](int r, int k) { const int i = i0 + r; return i < n ? W[k + n * i] : 0.0; },
                          [&](int r, int k) { const int j = j0 + r; return j < n ? W[k + n * j] : 0.0; },
                          i0, (int)n, acc, sm, NoFold{});
    double *T = P + ((int64_t)blockIdx.x * (blockIdx.x + 1) / 2 + blockIdx.y) * kTileB * kTileB;
    each_out(acc, [&](int r, int c, double v) { T[c * kTileB + r] = v; });
}

// One level of the bottom-up block inversion of a lower-triangular L (n x n):
// node z covers rows [r0, r0 + 2 hs), r0 = 2 hs z, split at rh = r0 + hs; its
// two products, over blockIdx.z:
//   step 0:  T = L21 W11      (T stored where W21 goes in Tb)
//   step 1:  W21 = -W22 T
// W11 and W22 are complete from the level below.
__global__ void __launch_bounds__(kTileThreads)
inv_level_kernel(const double *__restrict__ L, double *__restrict__ W, double *__restrict__ Tb, int64_t n, int hs, int step)
{
    const int64_t r0 = (int64_t)blockIdx.z * 2 * hs, rh = r0 + hs;
    if (rh >= n) return;
    const int64_t r1 = r0 + 2 * hs < n ? r0 + 2 * hs : n;
    const int s2 = (int)(r1 - rh);
    if ((int)blockIdx.x * kTileB >= s2 || (int)blockIdx.y * kTileB >= hs) return;
    __shared__ double sm[tile_smem_vals<false, true>];
    const int i0 = blockIdx.x * kTileB, j0 = blockIdx.y * kTileB;
    // step 0: a(i,k) = L[rh+i][r0+k], b(j,k) = W[r0+k][r0+j], K = hs (W11 lower: k >= j)
    // step 1: a(i,k) = W[rh+i][rh+k], b(j,k) = T[rh+k][r0+j], K = s2 (W22 lower: k <= i)
    const int K = step == 0 ? hs : s2;
    const int kBeg = step == 0 ? (j0 / kTileK) * kTileK : 0;
    const int kEnd = step == 0 ? K : (i0 + kTileB < K ? i0 + kTileB : K);
    const double *A = step == 0 ? L + rh + n * r0 : W + rh + n * rh;
    const double *B = step == 0 ? W + r0 + n * r0 : Tb + rh + n * r0;
    double acc[4][4][2];
    zero_acc(acc);
    dmma_tile<false, true>([&](int r, int k) { const int i = i0 + r; return i < s2 ? A[i + n * k] : 0.0; },
                           [&](int r, int k) { const int j = j0 + r; return j < hs ? B[k + n * j] : 0.0; },
                           kBeg, kEnd, acc, sm, NoFold{});
    double *C = step == 0 ? Tb : W;
    each_out(acc, [&](int r, int c, double v) {
        const int i = i0 + r, j = j0 + c;
        if (i < s2 && j < hs) C[(rh + i) + n * (r0 + j)] = step == 0 ? v : -v;
    });
}

// ---- factorisation ----------------------------------------------------------------
// One warp factors the 32 x 32 block S (column-major, stride ld, lower part
// read and overwritten by L) with lane r holding row r: a[i] is entry
// (r, j + i) while column j is eliminated, so the loop body is the same for
// every column and stays in the instruction cache (the fully unrolled form was
// bound by instruction fetch: 42 us cold against 16.8 us repeated).  A second
// warp follows column by column with W = L^-1, lane c solving L w = e_c, so
// the inversion hides behind the pivots' square roots and divisions, whose
// latency bounds the block.  status: set when a pivot is not positive (the
// pivot is then taken as 1).  Called by 64 threads (warps 0 and 1).
constexpr int kCholLd = kDb + 2;         // column j of L from row j + 1 on: sL[j][i] = L[j + 1 + i][j]
__device__ __forceinline__ void chol_block_warps(double *S, int ld, double (*sL)[kCholLd], double *sInv, double *Ds, int ldd, int *status)
{
    const int r = threadIdx.x & 31;
    if (threadIdx.x < 32) {
        double a[kDb];
#pragma unroll
        for (int c = 0; c < kDb; ++c) a[c] = c <= r ? S[r + ld * c] : 0.0;
#pragma unroll 1
        for (int j = 0; j < kDb; ++j) {
            double d = __shfl_sync(0xffffffffu, a[0], j);
            if (!(d > 0.0)) { if (r == j) atomicExch(status, 1); d = 1.0; }
            const double ljj = sqrt(d), rl = 1.0 / ljj;
            const double l = r == j ? ljj : a[0] * rl;       // rows above j hold leftovers that nothing reads
            if (r > j) sL[j][r - j - 1] = l;
            if (r == j) sInv[j] = rl;
            if (r >= j) S[r + ld * j] = l;
            asm volatile("bar.sync 1, 64;" ::: "memory");    // column j to both warps
#pragma unroll
            for (int i = 1; i < kDb; i += 2) {
                // past the block's last column: leftovers, never read back
                const double2 lc = *reinterpret_cast<const double2 *>(&sL[j][i - 1]);
                a[i - 1] = fma(-l, lc.x, a[i]);
                if (i + 1 < kDb) a[i] = fma(-l, lc.y, a[i + 1]);
            }
        }
    } else {
        double w[kDb];                   // w[i] = entry (j + i, c) of W at step j
#pragma unroll
        for (int i = 0; i < kDb; ++i) w[i] = i == r ? 1.0 : 0.0;
#pragma unroll 1
        for (int j = 0; j < kDb; ++j) {
            asm volatile("bar.sync 1, 64;" ::: "memory");
            const double x = w[0] * sInv[j];
            Ds[j + ldd * r] = x;
#pragma unroll
            for (int i = 1; i < kDb; i += 2) {
                const double2 lc = *reinterpret_cast<const double2 *>(&sL[j][i - 1]);
                w[i - 1] = fma(-lc.x, x, w[i]);
                if (i + 1 < kDb) w[i] = fma(-lc.y, x, w[i + 1]);
            }
        }
    }
}
// 8 x 32 outputs by one warp from shared memory: acc[J] += sum_{k < 32}
// a(row g, k) b(col, k), a at Ap[row + lda k], b at Bp[col + ldb k]
__device__ __forceinline__ void dmma_8x32(const double *Ap, int lda, const double *Bp, int ldb, double (&acc)[4][2])
{
    const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
#pragma unroll
    for (int J = 0; J < 4; ++J) acc[J][0] = acc[J][1] = 0.0;
#pragma unroll
    for (int kk = 0; kk < kDb; kk += 4) {
        const double a = Ap[g + lda * (kk + q)];
#pragma unroll
        for (int J = 0; J < 4; ++J) dmma_8x8x4(acc[J][0], acc[J][1], a, Bp[8 * J + g + ldb * (kk + q)]);
    }
}
// the warp's 8 x 32 outputs into column-major Sp (stride ld): assigned, or subtracted
__device__ __forceinline__ void put_8x32(double *Sp, int ld, const double (&acc)[4][2], bool subtract)
{
    const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
#pragma unroll
    for (int J = 0; J < 4; ++J)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            double *p = Sp + g + ld * (8 * J + 2 * q + h);
            *p = subtract ? *p - acc[J][h] : acc[J][h];
        }
}

constexpr int kDiagLd = kPb + 4, kDiagThreads = 256;
constexpr size_t kDiagSmem = sizeof(double) * (kPb * kDiagLd + kDb * kCholLd + kDb + kDb * 36);
// The 128 x 128 diagonal block at column k0 in one CTA: L over A's lower part,
// the 32 x 32 diagonal blocks' inverses to Dinv (rows / columns past n the identity).
__global__ void __launch_bounds__(kDiagThreads)
chol_diag_kernel(double *A, int64_t n, int64_t k0, double *Dinv, int *status)
{
    extern __shared__ __align__(16) double dsm[];
    double *S = dsm;                                                     // [128 columns][132]
    double (*sL)[kCholLd] = reinterpret_cast<double (*)[kCholLd]>(dsm + kPb * kDiagLd);
    double *sInv = dsm + kPb * kDiagLd + kDb * kCholLd, *Ds = sInv + kDb;    // Ds: [32 columns][36]
    const int t = threadIdx.x, warp = t >> 5;
    const int wb = n - k0 < kPb ? (int)(n - k0) : kPb, nb = (wb + kDb - 1) / kDb;
#pragma unroll 16
    for (int u = 0; u < kPb * kPb / kDiagThreads; ++u) {                 // 16 loads in flight
        const int e = t + u * kDiagThreads, i = e % kPb, c = e / kPb;
        S[i + kDiagLd * c] = (i < wb && c <= i) ? A[(k0 + i) + n * (k0 + c)] : (i == c ? 1.0 : 0.0);
    }
    __syncthreads();
    for (int b = 0; b < nb; ++b) {
        const int c0 = kDb * b;
        if (t < 64) chol_block_warps(S + c0 + kDiagLd * c0, kDiagLd, sL, sInv, Ds, 36, status);
        __syncthreads();
        for (int e = t; e < kDb * kDb; e += kDiagThreads) Dinv[(k0 / kDb + b) * kDb * kDb + e] = Ds[e % kDb + 36 * (e / kDb)];
        // rows below the block: L = A D^T, eight rows a warp at a time
        for (int r = c0 + kDb + 8 * warp; r < kDb * nb; r += kDiagThreads / 4) {
            double acc[4][2];
            dmma_8x32(S + r + kDiagLd * c0, kDiagLd, Ds, 36, acc);
            __syncwarp();
            put_8x32(S + r + kDiagLd * c0, kDiagLd, acc, false);
        }
        __syncthreads();
        // the later columns' rank-32 update
        for (int b2 = b + 1; b2 < nb; ++b2)
            for (int r = kDb * b2 + 8 * warp; r < kDb * nb; r += kDiagThreads / 4) {
                double acc[4][2];
                dmma_8x32(S + r + kDiagLd * c0, kDiagLd, S + kDb * b2 + kDiagLd * c0, kDiagLd, acc);
                put_8x32(S + r + kDiagLd * kDb * b2, kDiagLd, acc, true);
            }
        __syncthreads();
    }
    for (int e = t; e < kPb * kPb; e += kDiagThreads) {
        const int i = e % kPb, c = e / kPb;
        if (i < wb && c <= i) A[(k0 + i) + n * (k0 + c)] = S[i + kDiagLd * c];
    }
}
// The panel below a full 128-column diagonal block: 64 rows a CTA in shared
// memory, block by block L_b = A_b D_b^T and A_b2 -= L_b L11(b2, b)^T for the
// blocks b2 to its right.
constexpr int kPanelLd = kTileB + 4;
constexpr size_t kPanelSmem = sizeof(double) * (kPb * kPanelLd + 10 * kDb * 36);
constexpr int kPanelThreads = 256;
__global__ void __launch_bounds__(kPanelThreads)
chol_panel_kernel(double *A, int64_t n, int64_t k0, const double *__restrict__ Dinv)
{
    extern __shared__ __align__(16) double psm[];
    double *S = psm, *Bl = psm + kPb * kPanelLd;         // Bl: D_0..D_3, then L11(b2, b) for b < b2
    const int t = threadIdx.x, warp = t >> 5;
    const int64_t i0 = k0 + kPb + (int64_t)blockIdx.x * kTileB;
    const bool full = i0 + kTileB <= n;
#pragma unroll 16
    for (int u = 0; u < kTileB * kPb / kPanelThreads; ++u) {             // 16 loads in flight
        const int e = t + u * kPanelThreads, i = e % kTileB, c = e / kTileB;
        S[i + kPanelLd * c] = full || i0 + i < n ? A[(i0 + i) + n * (k0 + c)] : 0.0;
    }
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
        for (int u = 0; u < kDb * kDb / kPanelThreads; ++u) {
            const int e = t + u * kPanelThreads;
            Bl[b * kDb * 36 + e % kDb + 36 * (e / kDb)] = Dinv[(k0 / kDb + b) * kDb * kDb + e];
        }
#pragma unroll
    for (int b2 = 1; b2 < 4; ++b2)
#pragma unroll
        for (int b = 0; b < b2; ++b)
#pragma unroll
            for (int u = 0; u < kDb * kDb / kPanelThreads; ++u) {
                const int e = t + u * kPanelThreads;
                Bl[(4 + b2 * (b2 - 1) / 2 + b) * kDb * 36 + e % kDb + 36 * (e / kDb)] = A[(k0 + kDb * b2 + e % kDb) + n * (k0 + kDb * b + e / kDb)];
            }
    __syncthreads();
    // a warp's eight rows are its own from here on: no CTA-wide barrier
    double *R = S + 8 * warp;
    for (int b = 0; b < 4; ++b) {
        double acc[4][2];
        dmma_8x32(R + kPanelLd * kDb * b, kPanelLd, Bl + b * kDb * 36, 36, acc);
        __syncwarp();
        put_8x32(R + kPanelLd * kDb * b, kPanelLd, acc, false);
        __syncwarp();
        for (int b2 = b + 1; b2 < 4; ++b2) {
            dmma_8x32(R + kPanelLd * kDb * b, kPanelLd, Bl + (4 + b2 * (b2 - 1) / 2 + b) * kDb * 36, 36, acc);
            put_8x32(R + kPanelLd * kDb * b2, kPanelLd, acc, true);
        }
        __syncwarp();
    }
    __syncthreads();
    for (int e = t; e < kTileB * kPb; e += kPanelThreads) {
        const int i = e % kTileB, c = e / kTileB;
        if (i0 + i < n) A[(i0 + i) + n * (k0 + c)] = S[i + kPanelLd * c];
    }
}
// A22 -= L21 L21^T on the lower tiles of the trailing matrix (first row and
// column k0 + 128) from tile column jt on, the step's four blocks one after
// another: the tile stays in registers, so the trailing matrix is read and
// written once a step instead of once a block.
__global__ void __launch_bounds__(kTileThreads)
chol_trail_kernel(double *A, int64_t n, int64_t k0, int jt)
{
    __shared__ double sm[tile_smem_vals<false, false>];
    const int i0 = blockIdx.x * kTileB, j0 = (blockIdx.y + jt) * kTileB;
    if (j0 > i0) return;
    const int64_t t0 = k0 + kPb;
    const int m = (int)(n - t0);
    const double *L = A + t0 + n * k0;
    double *C = A + t0 * (1 + n);
    double acc[4][4][2], c[4][4][2];
    zero_acc(acc);
    each_out(c, [&](int r, int col, double &v) { const int i = i0 + r, j = j0 + col; v = (i < m && j < m) ? C[i + n * j] : 0.0; });
    dmma_tile<false, false>([&](int r, int k) { const int i = i0 + r; return i < m ? L[i + n * k] : 0.0; },
                            [&](int r, int k) { const int j = j0 + r; return j < m ? L[j + n * k] : 0.0; },
                            0, kPb, acc, sm, [&] {
#pragma unroll
        for (int I = 0; I < 4; ++I)
#pragma unroll
            for (int J = 0; J < 4; ++J)
#pragma unroll
                for (int h = 0; h < 2; ++h) { c[I][J][h] -= acc[I][J][h]; acc[I][J][h] = 0.0; }
    });
    each_out(c, [&](int r, int col, double &v) { const int i = i0 + r, j = j0 + col; if (i < m && j < m) C[i + n * j] = v; });
}

// copy the diagonal blocks' inverses into W's diagonal blocks (upper parts zero)
__global__ void place_dinv_kernel(const double *__restrict__ Dinv, double *__restrict__ W, int64_t n)
{
    const int64_t b = blockIdx.x;
    const int r = threadIdx.x % kDb, c = threadIdx.x / kDb;      // 32 x 32 threads
    const int64_t i = b * kDb + r, j = b * kDb + c;
    if (i < n && j < n) W[i + n * j] = Dinv[b * kDb * kDb + r + kDb * c];
}

}  // namespace topgpu
