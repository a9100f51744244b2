// topgpu_dense.cuh -- dense FP64 linear algebra of the coarsest level: the
// Cholesky factor of the assembled coarsest matrix and its explicit inverse
// (the V-cycle's coarsest solve is one GEMV with it).
//
//   * factorisation: right-looking over 32-column blocks, taken 128 columns at
//     a time: chol_diag_kernel factors the 128 x 128 diagonal block in one
//     CTA's shared memory (and inverts its four 32 x 32 diagonal blocks),
//     chol_panel_kernel forms the panel below it, L21 = A21 L11^-T block by
//     block, and chol_next_kernel (the next step's columns) and chol_trail_kernel
//     (the others) apply the four rank-32 updates A22 -= L21 L21^T to every
//     trailing tile in one pass.  Each entry still
//     receives the 32-column blocks' contributions one after another, each
//     summed from zero, as a sweep of one block at a time gives them;
//   * W = L^-1 by 2x2 block inversion, [L11 0; L21 L22]^-1 =
//     [W11 0; -W22 L21 W11  W22], bottom-up from the factorisation's
//     diagonal blocks, each node as soon as its columns of L are complete, or
//     after the factor every node of a level in one launch;
//   * A^-1 = W^T W on the lower tiles, mirrored, skipping the zero blocks of W.
//
// Measured on one B200, factor and inverse (bit-identical to the sweep of one
// 32-column block a step on SIMT tiles that this replaces): n = 336 506 -> 265
// us, n = 1386 2.31 -> 1.07 ms, n = 4131 12.4 -> 5.35 ms (the last factor and
// trailing updates 3.0 ms, W 1.4 ms, W^T W 0.9 ms; its 35 G multiply-adds take
// 2.5 ms at the FP64 peak).  Small sizes are bound by the chain diagonal block ->
// panel -> next columns, 37 + 8 + 6..8 us a step of 128 columns at n = 1386
// (one warp a block, panels of 64 rows a CTA, 64 x 64 tiles throughout: 49 + 15
// + 13 us), and that by the pivots' square roots and reciprocals (below).
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
#include <algorithm>
#include <cstdint>
#include "topgpu_kernels.cuh"
#include "topgpu_grid.cuh"
#include "topgpu_streams.h"

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
// two products, over blockIdx.z from node z0 on:
//   step 0:  T = L21 W11      (T stored where W21 goes in Tb)
//   step 1:  W21 = -W22 T
// W11 and W22 are complete from the level below.
__global__ void __launch_bounds__(kTileThreads)
inv_level_kernel(const double *__restrict__ L, double *__restrict__ W, double *__restrict__ Tb, int64_t n, int hs, int step, int z0)
{
    const int64_t r0 = (int64_t)(z0 + blockIdx.z) * 2 * hs, rh = r0 + hs;
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
// Six warps factor the 32 x 32 block S (column-major, stride ld, lower part read
// and overwritten by L, upper part by leftovers) and invert it.  Warp w < 4 holds
// columns 8 w .. 8 w + 7, lane r row r, and eliminates with its columns while the
// later ones follow; warps 4 and 5 follow with W = L^-1, solving L w = e_c, two lanes a
// column (even and odd rows).  What
// bounds the block is the chain pivot -> square root -> reciprocal -> column -> next
// pivot (104 + 75 cycles for the first two, 23 a multiply-add, 27 a shuffle).  So
// the lane of the next row forms its pivot from its own entries before the column
// goes to shared memory, a column's owner has at most seven updates to issue, and it
// tells the others on the column's own mbarrier (ready[j], one phase a block; no
// cycles lost on the chain, where a barrier they all meet at cost 70 a column).
// a[i] is entry (r, j + i) while the owner eliminates column j, so the loop body is
// the same for every column and stays in the instruction cache.  status: kCholPivot
// is set when a pivot is not positive (the pivot is then taken as 1), kCholWait
// when a wait for a column ran out.
constexpr int kCholPivot = 1, kCholWait = 2;
constexpr int kCholLd = kDb + 2;         // column j of L from row j + 1 on: sL[j][i] = L[j + 1 + i][j]
constexpr int kCholWarps = 6;
__device__ __forceinline__ void chol_ready(uint64_t *ready)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" :: "r"((unsigned)__cvta_generic_to_shared(ready)) : "memory");
}
// Bounded (one second): past it the status says so, the warp goes on, and waits
// that do not end at once give up from then on.  The clock and the status are
// looked at every 64th try, so a wait that ends costs its tries alone.
__device__ __forceinline__ void chol_await(uint64_t *ready, int phase, int *status)
{
    const unsigned a = (unsigned)__cvta_generic_to_shared(ready);
    auto over = [&] {
        unsigned ok;
        asm volatile("{.reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p;}" : "=r"(ok) : "r"(a), "r"(phase) : "memory");
        return ok != 0;
    };
    if (over()) return;
    const uint64_t t0 = bulk::now_ns();
    for (unsigned tries = 1; !over(); ++tries)
        if (tries % 64 == 0 && ((*(volatile int *)status & kCholWait) || bulk::now_ns() - t0 > bulk::kWaitNs)) {
            atomicOr(status, kCholWait);
            return;
        }
}
__device__ __forceinline__ void chol_block_warps(int w, double *S, int ld, double (*sL)[kCholLd], double *sInv, double *Ds, int ldd, uint64_t *ready, int phase, int *status)
{
    const int r = threadIdx.x & 31;
    if (w < 4) {
        double a[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) a[i] = 8 * w + i <= r ? S[r + ld * (8 * w + i)] : 0.0;
#pragma unroll 1
        for (int j = 0; j < 8 * w; ++j) {                        // earlier owners' columns
            chol_await(ready + j, phase, status);
            const double l = S[r + ld * j];
#pragma unroll
            for (int i = 0; i < 8; i += 2) {
                const double2 lc = *reinterpret_cast<const double2 *>(S + ld * j + 8 * w + i);
                a[i] = fma(-l, lc.x, a[i]);
                a[i + 1] = fma(-l, lc.y, a[i + 1]);
            }
        }
        double d = __shfl_sync(0xffffffffu, a[0], 8 * w);
        bool bad = false;
#pragma unroll 1
        for (int j = 8 * w; j < 8 * w + 8; ++j) {
            const bool ok = d > 0.0;                             // beside the root: a test ahead of it cost 85 cycles a column
            const double root = sqrt(d), inv = 1.0 / root;
            const double ljj = ok ? root : 1.0, rl = ok ? inv : 1.0;
            bad = bad || !ok;
            const double l = a[0] * rl;                          // rows above j hold leftovers that nothing uses
            d = __shfl_sync(0xffffffffu, fma(-l, l, a[1]), j + 1);     // the next pivot; past the segment: not used
            const double lj = r == j ? ljj : l;
            sL[j][(r - j - 1) & 31] = lj;
            sInv[j] = rl;
            S[r + ld * j] = lj;
            __syncwarp();
            if (r == 0) chol_ready(ready + j);
#pragma unroll
            for (int i = 1; i < 8; i += 2) {
                // past the warp's last column: leftovers, never read back
                const double2 lc = *reinterpret_cast<const double2 *>(&sL[j][i - 1]);
                a[i - 1] = fma(-l, lc.x, a[i]);
                if (i + 1 < 8) a[i] = fma(-l, lc.y, a[i + 1]);
            }
        }
        if (bad && r == 0) atomicOr(status, kCholPivot);
    } else {
        const int h = r >> 4, c = (r & 15) + 16 * (w - 4);
        double x[kDb / 2];               // x[i] = entry (j + 2 i + h, c) of W at even steps j
#pragma unroll
        for (int i = 0; i < kDb / 2; ++i) x[i] = 2 * i + h == c ? 1.0 : 0.0;
#pragma unroll 1
        for (int j = 0; j < kDb; j += 2) {
            chol_await(ready + j, phase, status);
            const double y0 = __shfl_sync(0xffffffffu, x[0] * sInv[j], r & 15);
            // row j + 2 i + h: L[row][j] = sL[j][row - j - 1] (i = 0 of the even half is row j itself: not used again)
#pragma unroll
            for (int i = 0; i < kDb / 2; ++i) x[i] = fma(-sL[j][i || h ? 2 * i + h - 1 : 0], y0, x[i]);
            chol_await(ready + j + 1, phase, status);
            const double y1 = __shfl_sync(0xffffffffu, x[0] * sInv[j + 1], (r & 15) + 16);
            Ds[j + h + ldd * c] = h ? y1 : y0;
            // row j + 2 i + h of the next pair, i from 1: sL[j + 1][row - j - 2]
#pragma unroll
            for (int i = 1; i < kDb / 2; ++i) x[i - 1] = fma(-sL[j + 1][2 * i + h - 2], y1, x[i]);
        }
    }
}
// 8 x 8 NJ outputs by one warp from shared memory: acc[J] = sum_{k < 32}
// a(row g, k) b(col, k), a at Ap[row + lda k], b at Bp[col + ldb k]
template <int NJ>
__device__ __forceinline__ void dmma_8x(const double *Ap, int lda, const double *Bp, int ldb, double (&acc)[NJ][2])
{
    const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
#pragma unroll
    for (int J = 0; J < NJ; ++J) acc[J][0] = acc[J][1] = 0.0;
#pragma unroll
    for (int kk = 0; kk < kDb; kk += 4) {
        const double a = Ap[g + lda * (kk + q)];
#pragma unroll
        for (int J = 0; J < NJ; ++J) dmma_8x8x4(acc[J][0], acc[J][1], a, Bp[8 * J + g + ldb * (kk + q)]);
    }
}
// the warp's 8 x 8 NJ outputs into column-major Sp (stride ld): assigned, or subtracted
template <int NJ>
__device__ __forceinline__ void put_8x(double *Sp, int ld, const double (&acc)[NJ][2], bool subtract)
{
    const int lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
#pragma unroll
    for (int J = 0; J < NJ; ++J)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            double *p = Sp + g + ld * (8 * J + 2 * q + h);
            *p = subtract ? *p - acc[J][h] : acc[J][h];
        }
}

constexpr int kDiagLd = kPb + 4, kDiagThreads = 512;
constexpr size_t kDiagSmem = sizeof(double) * (kPb * kDiagLd + kDb * kCholLd + kDb + 2 * kDb * 36) + sizeof(uint64_t) * kDb;
// The 128 x 128 diagonal block at column k0 in one CTA, 37 us: four 32-column blocks of
// about 11,700 cycles (their chain), the products between them 18,000 cycles at
// one SM's FP64 rate.  L over A's lower part,
// the 32 x 32 diagonal blocks' inverses to Dinv (rows / columns past n the identity).
// Between two 32-column blocks only the next diagonal block is brought up to
// date; the other updates are the remaining warps' while six factor it.
__global__ void __launch_bounds__(kDiagThreads)
chol_diag_kernel(double *A, int64_t n, int64_t k0, double *Dinv, int *status)
{
    extern __shared__ __align__(16) double dsm[];
    double *S = dsm;                                                     // [128 columns][132]
    double (*sL)[kCholLd] = reinterpret_cast<double (*)[kCholLd]>(dsm + kPb * kDiagLd);
    double *sInv = dsm + kPb * kDiagLd + kDb * kCholLd, *DsAll = sInv + kDb;    // two of [32 columns][36]
    uint64_t *ready = reinterpret_cast<uint64_t *>(DsAll + 2 * kDb * 36);
    const int t = threadIdx.x, warp = t >> 5;
    constexpr int rest = kDiagThreads / 32 - kCholWarps;                 // warps beside the factorising ones
    const int idle = warp - kCholWarps;                                  // their index among those
    const int wb = n - k0 < kPb ? (int)(n - k0) : kPb, nb = (wb + kDb - 1) / kDb;
    if (t < kDb) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"((unsigned)__cvta_generic_to_shared(ready + t)) : "memory");
    if (wb == kPb) {                     // the whole square, sixteen loads in flight; its upper part is cleared here
        const double *a = A + k0 + (t & (kPb - 1)) + n * (k0 + t / kPb);
        const int i = t & (kPb - 1);
#pragma unroll 16
        for (int u = 0; u < kPb * kPb / kDiagThreads; ++u) {
            const int c = t / kPb + u * (kDiagThreads / kPb);
            const double v = a[n * (u * (kDiagThreads / kPb))];
            S[i + kDiagLd * c] = c <= i ? v : 0.0;
        }
    } else {
        for (int e = t; e < kPb * kPb; e += kDiagThreads) {
            const int i = e % kPb, c = e / kPb;
            S[i + kDiagLd * c] = (i < wb && c <= i) ? A[(k0 + i) + n * (k0 + c)] : (i == c ? 1.0 : 0.0);
        }
    }
    __syncthreads();
    auto put_columns = [&](int b, int t0, int step) {                    // block b's columns of L
        const int h = kPb - kDb * b;
        for (int e = t0; e < kDb * h; e += step) {
            const int c = kDb * b + e / h, i = kDb * b + e % h;
            if (i < wb && c <= i) A[(k0 + i) + n * (k0 + c)] = S[i + kDiagLd * c];
        }
    };
    for (int b = 0; b < nb; ++b) {
        const int c0 = kDb * b, p0 = c0 - kDb;
        double *Ds = DsAll + (b & 1) * kDb * 36;
        if (warp < kCholWarps) {
            if (b) {                     // the block's own update by the last block's columns
                if (warp < 4) {
                    double acc[4][2];
                    const int r = c0 + 8 * warp;
                    dmma_8x(S + r + kDiagLd * p0, kDiagLd, S + c0 + kDiagLd * p0, kDiagLd, acc);
                    put_8x(S + r + kDiagLd * c0, kDiagLd, acc, true);
                }
                asm volatile("bar.sync 1, %0;" :: "n"(32 * kCholWarps) : "memory");
            }
            chol_block_warps(warp, S + c0 + kDiagLd * c0, kDiagLd, sL, sInv, Ds, 36, ready, b & 1, status);
        } else if (b) {
            // the other entries' update by the last block's columns, and its inverse
            int item = 0;
            for (int b2 = b; b2 < nb; ++b2)
                for (int r = kDb * b2 + (b2 == b ? kDb : 0); r < kDb * nb; r += 8) {
                    if (item++ % rest != idle) continue;
                    double acc[4][2];
                    dmma_8x(S + r + kDiagLd * p0, kDiagLd, S + kDb * b2 + kDiagLd * p0, kDiagLd, acc);
                    put_8x(S + r + kDiagLd * kDb * b2, kDiagLd, acc, true);
                }
            const double *Dp = DsAll + ((b - 1) & 1) * kDb * 36;
            const int ti = 32 * idle + (t & 31);
            put_columns(b - 1, ti, 32 * rest);
            for (int e = ti; e < kDb * kDb; e += 32 * rest) Dinv[(k0 / kDb + b - 1) * kDb * kDb + e] = Dp[e % kDb + 36 * (e / kDb)];
        }
        __syncthreads();
        // rows below the block: L = A D^T, eight rows a warp
        for (int r = c0 + kDb + 8 * warp; r < kDb * nb; r += kDiagThreads / 4) {
            double acc[4][2];
            dmma_8x(S + r + kDiagLd * c0, kDiagLd, Ds, 36, acc);
            __syncwarp();
            put_8x(S + r + kDiagLd * c0, kDiagLd, acc, false);
        }
        __syncthreads();
    }
    for (int e = t; e < kDb * kDb; e += kDiagThreads)
        Dinv[(k0 / kDb + nb - 1) * kDb * kDb + e] = DsAll[((nb - 1) & 1) * kDb * 36 + e % kDb + 36 * (e / kDb)];
    put_columns(nb - 1, t, kDiagThreads);
}
// The panel below a full 128-column diagonal block: R rows a CTA in shared
// memory, block by block L_b = A_b D_b^T and A_b2 -= L_b L11(b2, b)^T for the
// blocks b2 to its right.  Eight warps, each eight rows by R / 2 columns of a
// block: the fewer rows a CTA has, the shorter its chain of ten products, which is
// what a panel that leaves the chip idle waits for (the products' rate on one SM).
constexpr int kPanelThreads = 256;
template <int R> constexpr size_t kPanelSmem = sizeof(double) * (kPb * (R + 4) + 10 * kDb * 36);
template <int R>
__global__ void __launch_bounds__(kPanelThreads)
chol_panel_kernel(double *A, int64_t n, int64_t k0, const double *__restrict__ Dinv)
{
    constexpr int ld = R + 4, J = R / 16;                // J 8-column tiles a warp
    extern __shared__ __align__(16) double psm[];
    double *S = psm, *Bl = psm + kPb * ld;               // Bl: D_0..D_3, then L11(b2, b) for b < b2
    const int t = threadIdx.x, warp = t >> 5;
    const int64_t i0 = k0 + kPb + (int64_t)blockIdx.x * R;
    const bool full = i0 + R <= n;
#pragma unroll 16
    for (int u = 0; u < R * kPb / kPanelThreads; ++u) {                  // 16 loads in flight
        const int e = t + u * kPanelThreads, i = e % R, c = e / R;
        S[i + ld * c] = full || i0 + i < n ? A[(i0 + i) + n * (k0 + c)] : 0.0;
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
    // with all 32 columns a warp's eight rows are its own from here on: no CTA-wide barrier
    auto meet = [] { if (J == 4) __syncwarp(); else __syncthreads(); };
    double *Rw = S + 8 * (warp % (R / 8));
    const int cw = (warp / (R / 8)) * (8 * J);           // the warp's first column in a block
    for (int b = 0; b < 4; ++b) {
        double acc[J][2];
        dmma_8x(Rw + ld * kDb * b, ld, Bl + b * kDb * 36 + cw, 36, acc);
        meet();
        put_8x(Rw + ld * (kDb * b + cw), ld, acc, false);
        meet();
        for (int b2 = b + 1; b2 < 4; ++b2) {
            dmma_8x(Rw + ld * kDb * b, ld, Bl + (4 + b2 * (b2 - 1) / 2 + b) * kDb * 36 + cw, 36, acc);
            put_8x(Rw + ld * (kDb * b2 + cw), ld, acc, true);
        }
        meet();
    }
    __syncthreads();
    for (int e = t; e < R * kPb; e += kPanelThreads) {
        const int i = e % R, c = e / R;
        if (i0 + i < n) A[(i0 + i) + n * (k0 + c)] = S[i + ld * c];
    }
}
// Its launch for the rows below column k0 + 128 on st: the fewest rows a CTA that
// still make one wave of the SMs.
inline void chol_panel(double *A, int64_t n, int64_t k0, const double *Dinv, int sms, cudaStream_t st)
{
    const int64_t rest = n - k0 - kPb;
    auto ctas = [&](int R) { return (unsigned)((rest + R - 1) / R); };
    if (ctas(16) <= (unsigned)sms) chol_panel_kernel<16><<<ctas(16), kPanelThreads, kPanelSmem<16>, st>>>(A, n, k0, Dinv);
    else if (ctas(32) <= (unsigned)sms) chol_panel_kernel<32><<<ctas(32), kPanelThreads, kPanelSmem<32>, st>>>(A, n, k0, Dinv);
    else chol_panel_kernel<64><<<ctas(64), kPanelThreads, kPanelSmem<64>, st>>>(A, n, k0, Dinv);
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

// The same update of the next step's 128 columns alone, ahead of the others: what the
// next diagonal block waits for.  32 x 32 outputs a CTA with both operands' 128
// columns in shared memory at once: a short chain on many SMs, where the 64 x 64
// tiles of the kernel above take four times the products an SM.
constexpr int kNextThreads = 256, kNextLd = kDb + 4;
constexpr size_t kNextSmem = sizeof(double) * 2 * kPb * kNextLd;
__global__ void __launch_bounds__(kNextThreads)
chol_next_kernel(double *A, int64_t n, int64_t k0)
{
    extern __shared__ __align__(16) double nsm[];
    double *Li = nsm, *Lj = nsm + kPb * kNextLd;
    const int i0 = blockIdx.x * kDb, j0 = blockIdx.y * kDb;
    if (j0 > i0) return;
    const int t = threadIdx.x, warp = t >> 5, g = (t & 31) >> 2, q = t & 3;
    const int64_t t0 = k0 + kPb;
    const int m = (int)(n - t0);
    const double *L = A + t0 + n * k0;
    double *C = A + t0 * (1 + n);
    const int r0 = 8 * (warp & 3), c0 = 16 * (warp >> 2);                // the warp's 8 x 16 outputs
    double c[2][2], acc[2][2];
#pragma unroll
    for (int J = 0; J < 2; ++J)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int i = i0 + r0 + g, j = j0 + c0 + 8 * J + 2 * q + h;
            c[J][h] = (i < m && j < m) ? C[i + n * j] : 0.0;
        }
#pragma unroll
    for (int u = 0; u < kDb * kPb / kNextThreads; ++u) {
        const int e = t + u * kNextThreads, r = e % kDb, k = e / kDb;
        Li[r + kNextLd * k] = i0 + r < m ? L[i0 + r + n * k] : 0.0;
        Lj[r + kNextLd * k] = j0 + r < m ? L[j0 + r + n * k] : 0.0;
    }
    __syncthreads();
#pragma unroll
    for (int b = 0; b < 4; ++b) {
        dmma_8x(Li + r0 + kNextLd * kDb * b, kNextLd, Lj + c0 + kNextLd * kDb * b, kNextLd, acc);
#pragma unroll
        for (int J = 0; J < 2; ++J)
#pragma unroll
            for (int h = 0; h < 2; ++h) c[J][h] -= acc[J][h];
    }
#pragma unroll
    for (int J = 0; J < 2; ++J)
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int i = i0 + r0 + g, j = j0 + c0 + 8 * J + 2 * q + h;
            if (i < m && j < m) C[i + n * j] = c[J][h];
        }
}
inline void chol_next(double *A, int64_t n, int64_t k0, cudaStream_t st)
{
    const int64_t rest = n - k0 - kPb, tiles = (rest + kDb - 1) / kDb;
    chol_next_kernel<<<dim3((unsigned)tiles, (unsigned)(tiles < 4 ? tiles : 4)), kNextThreads, kNextSmem, st>>>(A, n, k0);
}

// opts the factorisation's kernels into their shared memory
inline cudaError_t chol_smem_attr()
{
    cudaError_t e = cudaSuccess;
    auto opt = [&](auto kernel, size_t bytes) {
        if (e == cudaSuccess) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    };
    opt(chol_diag_kernel, kDiagSmem);
    opt(chol_panel_kernel<16>, kPanelSmem<16>);
    opt(chol_panel_kernel<32>, kPanelSmem<32>);
    opt(chol_panel_kernel<64>, kPanelSmem<64>);
    opt(chol_next_kernel, kNextSmem);
    return e;
}

// copy the diagonal blocks' inverses from block b0 on into W's diagonal blocks (upper parts zero)
__global__ void place_dinv_kernel(const double *__restrict__ Dinv, double *__restrict__ W, int64_t n, int64_t b0)
{
    const int64_t b = b0 + blockIdx.x;
    const int r = threadIdx.x % kDb, c = threadIdx.x / kDb;      // 32 x 32 threads
    const int64_t i = b * kDb + r, j = b * kDb + c;
    if (i < n && j < n) W[i + n * j] = Dinv[b * kDb * kDb + r + kDb * c];
}
// What columns c0 .. c - 1 of L add to W = L^-1 (W zero before the first; c0 a multiple
// of 128; L complete in its columns before c): of every level, the products T of the
// nodes whose left half, and W21 of the nodes that, end there.  Called after each step of
// the factorisation on a stream beside it, this leaves the last rows' products for
// after the factor; called once, for all columns, it takes each level in two launches.
// Returns the launches.
inline int inverse_columns(const double *L, double *W, double *T, const double *Dinv, int64_t n, int64_t c0, int64_t c, cudaStream_t st)
{
    int launches = 1;
    place_dinv_kernel<<<(unsigned)((c - c0 + kDb - 1) / kDb), kDb * kDb, 0, st>>>(Dinv, W, n, c0 / kDb);
    for (int64_t hs = kDb; hs < n; hs *= 2) {
        const int64_t all = (n - hs + 2 * hs - 1) / (2 * hs);                // nodes with rows on both sides of their split
        auto left = [&](int64_t e) { return e < hs ? 0 : std::min(all, (e - hs) / (2 * hs) + 1); };
        auto whole = [&](int64_t e) { return e >= n ? all : std::min(all, e / (2 * hs)); };
        const unsigned tiles = (unsigned)((hs + kTileB - 1) / kTileB);
        for (int step = 0; step < 2; ++step) {
            const int64_t z0 = step ? whole(c0) : left(c0), z1 = step ? whole(c) : left(c);
            if (z1 <= z0) continue;
            inv_level_kernel<<<dim3(tiles, tiles, (unsigned)(z1 - z0)), kTileThreads, 0, st>>>(L, W, T, n, (int)hs, step, (int)z0);
            ++launches;
        }
    }
    return launches;
}


// The factor of A (n x n, lower part) over A and W = L^-1, on st and (n > kPb) the
// streams of f; T: n x n scratch, Dinv: 32 x 32 values a block of 32 columns.  Each
// step's trailing update is split: the next step's 128 columns first, on st, then the
// rest on f.aux, beside the next diagonal block (one CTA, 37 us) and panel, which
// touch other columns.  beside: W follows on f.inv, which reads finished columns
// alone and writes W and T; else after the factor.  st has waited for all of it at
// the end.  Up to kBesideMaxDofs the steps' chain leaves the chip idle and W is
// formed beside it (assembly, n = 675 706 -> 669 us, n = 1386 1.10 -> 1.08 ms); where
// the trailing updates fill the chip it is slower (n = 4131 5.15 ms after the factor,
// 5.48 beside it).  Between 1386 and 4131 the line was not looked for; it lies
// nearer the size at which the gain had shrunk to 2 %.
constexpr int64_t kBesideMaxDofs = 2000;
inline cudaError_t factor_and_inverse(double *A, double *W, double *T, double *Dinv, int64_t n, int *status, int sms, bool beside,
                                      cudaStream_t st, const FactorStreams &f, int64_t &launches)
{
    cudaStream_t si = beside ? f.inv : st;
    cudaError_t err = cudaSuccess;
    auto ok = [&](cudaError_t e) { if (err == cudaSuccess) err = e; return err == cudaSuccess; };
    auto reached = [&](cudaStream_t other) {           // other waits for what st holds so far
        return ok(cudaEventRecord(f.go, st)) && ok(cudaStreamWaitEvent(other, f.go, 0));
    };
    if (beside && !reached(si)) return err;
    if (!ok(cudaMemsetAsync(W, 0, sizeof(double) * n * n, si))) return err;
    constexpr int kNext = kPb / kTileB;                // tile columns of the next step
    bool restRuns = false;
    for (int64_t k0 = 0; k0 < n; k0 += kPb) {
        chol_diag_kernel<<<1, kDiagThreads, kDiagSmem, st>>>(A, n, k0, Dinv, status);
        ++launches;
        const int64_t rest = n - k0 - kPb;
        const int nt = rest > 0 ? (int)((rest + kTileB - 1) / kTileB) : 0;
        if (rest > 0) {
            chol_panel(A, n, k0, Dinv, sms, st);
            ++launches;
        }
        if (beside && !reached(si)) return err;
        if (rest > 0) {
            if (nt > kNext && !reached(f.aux)) return err;
            if (restRuns && !ok(cudaStreamWaitEvent(st, f.auxDone, 0))) return err;      // the previous step's updates of these columns
            chol_next(A, n, k0, st);
            ++launches;
            restRuns = nt > kNext;
            if (restRuns) {
                chol_trail_kernel<<<dim3((unsigned)nt, (unsigned)(nt - kNext)), kTileThreads, 0, f.aux>>>(A, n, k0, kNext);
                ++launches;
                if (!ok(cudaEventRecord(f.auxDone, f.aux))) return err;
            }
        }
        if (beside) launches += inverse_columns(A, W, T, Dinv, n, k0, std::min(n, k0 + kPb), si);
    }
    if (!beside) launches += inverse_columns(A, W, T, Dinv, n, 0, n, st);
    if (beside && ok(cudaEventRecord(f.invDone, si))) ok(cudaStreamWaitEvent(st, f.invDone, 0));
    return err;
}

}  // namespace topgpu
