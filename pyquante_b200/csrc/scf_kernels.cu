// Dense SCF step kernels of the batched and device SCF loops (no
// counterpart in the reference, whose SCF diagonalises on the host):
//   * purify_step_kernel: one step of the canonical purification of Palser
//     and Manolopoulos (Phys. Rev. B 58, 12704 (1998)) for a batch of
//     matrices, given P, P^2 and P^3 (two library GEMMs before it):
//       c = tr(P^2 - P^3) / tr(P - P^2), clamped to [0, 1];
//       P' = ((1+c) P^2 - P^3) / c             for c >= 1/2,
//       P' = ((1-2c) P + (1+c) P^2 - P^3) / (1-c)  otherwise;
//     a matrix already idempotent to rounding (|tr(P - P^2)| < tol n) is
//     kept and flagged done.  One block per matrix: the traces by a block
//     reduction, then the update, in one launch (the elementwise form in
//     tensor operations takes some fifteen launches per step);
//   * purify_kernel: the whole purification of one matrix by one block, for
//     matrices that fit in shared memory twice: the symmetric part of F, its
//     Gershgorin bounds, the linear start and the steps, with P and P^2 kept in
//     shared memory and the products on FP64 tensor cores over the lower triangle;
//   * solve_small_kernel: the DIIS equations of a batch, one warp each.
#include <cmath>
#include <cstdint>

#include <cuda_runtime.h>

#include "../../include/pyquante_b200.h"
#include "dmma.cuh"

using namespace pqb;

namespace {

constexpr int kPurifyThreads = 256;

__global__ void __launch_bounds__(kPurifyThreads) purify_step_kernel(int n, const double *__restrict__ P,
                                                                   const double *__restrict__ P2,
                                                                   const double *__restrict__ P3,
                                                                   double *__restrict__ Pout, int *__restrict__ done,
                                                                   double tol)
{
    const int64_t off = (int64_t)blockIdx.x * n * n;
    const double *p = P + off, *p2 = P2 + off, *p3 = P3 + off;
    double *po = Pout + off;
    __shared__ double s_num[kPurifyThreads / 32], s_den[kPurifyThreads / 32];
    double num = 0.0, den = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const int64_t ii = (int64_t)i * n + i;
        num += p2[ii] - p3[ii];
        den += p[ii] - p2[ii];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        num += __shfl_xor_sync(0xffffffffu, num, o);
        den += __shfl_xor_sync(0xffffffffu, den, o);
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) {
        s_num[warp] = num;
        s_den[warp] = den;
    }
    __syncthreads();
    num = 0.0;
    den = 0.0;
#pragma unroll
    for (int w = 0; w < kPurifyThreads / 32; ++w) {
        num += s_num[w];
        den += s_den[w];
    }
    const bool fin = fabs(den) < tol * n;
    double c = fin ? 0.5 : num / den;
    c = c < 0.0 ? 0.0 : (c > 1.0 ? 1.0 : c);
    const bool hi = c >= 0.5;
    const double a0 = hi ? 0.0 : (1.0 - 2.0 * c), a1 = 1.0 + c;
    const double inv = 1.0 / (hi ? (c > 1e-300 ? c : 1e-300) : ((1.0 - c) > 1e-300 ? (1.0 - c) : 1e-300));
    const int64_t nn = (int64_t)n * n;
    for (int64_t e = threadIdx.x; e < nn; e += blockDim.x) {
        const double x = p[e];
        po[e] = fin ? x : fma(a0, x, fma(a1, p2[e], -p3[e])) * inv;
    }
    if (threadIdx.x == 0 && done) done[blockIdx.x] = fin ? 1 : 0;
}

// ---- the whole purification of a matrix of up to kPurifyMax rows.  16 warps
// share the 16 x 16 tiles of the lower triangle; tr P^3 = sum_ij (P^2)_ij P_ij
// gives the step's c before the second product, whose tiles stay in registers
// until every warp has read P.  Bound by the serial chain of steps, each two
// products with the block's tensor throughput.  A batch of 32 water clusters (n
// = 7 to 95, eight size buckets) takes 4.5 ms an SCF iteration, 8.4 ms with two
// library GEMMs and one update kernel per step, 48 steps whether needed or not.
constexpr int kPurifyMax = 112, kPurifyWarps = 16;
constexpr int kPurifyTiles = (kPurifyMax / 16) * (kPurifyMax / 16 + 1) / 2;
constexpr int kPurifyRounds = (kPurifyTiles + kPurifyWarps - 1) / kPurifyWarps;

__device__ __forceinline__ double block_sum(double x, double *red)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    __syncthreads();   // red is free again
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = x;
    __syncthreads();
    double s = 0.0;
#pragma unroll
    for (int w = 0; w < kPurifyWarps; ++w) s += red[w];
    return s;
}

// acc = the 16 x 16 tile (i0, j0) of X Y, both symmetric (Y's rows serve as its columns)
__device__ __forceinline__ void tile_product(const double *X, const double *Y, int pitch, int np, int i0, int j0, int lane,
                                             double (&acc)[2][2][2])
{
    const double *x = X + (i0 + (lane >> 2)) * pitch + (lane & 3), *y = Y + (j0 + (lane >> 2)) * pitch + (lane & 3);
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 2; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;
#pragma unroll 4
    for (int k = 0; k < np; k += 4) {
        const double x0 = x[k], x1 = x[8 * pitch + k], y0 = y[k], y1 = y[8 * pitch + k];
        dmma(acc[0][0], x0, y0);
        dmma(acc[0][1], x0, y1);
        dmma(acc[1][0], x1, y0);
        dmma(acc[1][1], x1, y1);
    }
}

__global__ void __launch_bounds__(kPurifyWarps * 32) purify_kernel(int n, const double *__restrict__ F,
                                                                   const double *__restrict__ nocc,
                                                                   const unsigned char *__restrict__ pad,
                                                                   double *__restrict__ Pout, int *__restrict__ done,
                                                                   int maxit, double tol)
{
    extern __shared__ double sm[];
    __shared__ double red[kPurifyWarps], s_hi[kPurifyWarps], s_lo[kPurifyWarps];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nt = (n + 15) / 16, np = 16 * nt, pitch = np + 4;
    double *P = sm, *P2 = sm + np * pitch;
    const double *f = F + (int64_t)blockIdx.x * n * n;
    const unsigned char *pd = pad ? pad + (int64_t)blockIdx.x * n : nullptr;
    for (int e = tid; e < 2 * np * pitch; e += blockDim.x) sm[e] = 0.0;
    __syncthreads();
    for (int e = tid; e < n * n; e += blockDim.x) {
        const int i = e / n, j = e - i * n;
        P[i * pitch + j] = 0.5 * (f[e] + f[j * n + i]);
    }
    __syncthreads();
    // Gershgorin bounds of the real rows; the padded ones go above them
    double hi = -1e300, lo = 1e300;
    if (tid < n && !(pd && pd[tid])) {
        double r = 0.0;
        for (int j = 0; j < n; ++j) r += fabs(P[tid * pitch + j]);
        const double d = P[tid * pitch + tid];
        r -= fabs(d);
        hi = d + r;
        lo = d - r;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double h = __shfl_xor_sync(0xffffffffu, hi, o), l = __shfl_xor_sync(0xffffffffu, lo, o);
        hi = h > hi ? h : hi;
        lo = l < lo ? l : lo;
    }
    if (lane == 0) {
        s_hi[warp] = hi;
        s_lo[warp] = lo;
    }
    __syncthreads();
#pragma unroll
    for (int w = 0; w < kPurifyWarps; ++w) {
        hi = s_hi[w] > hi ? s_hi[w] : hi;
        lo = s_lo[w] < lo ? s_lo[w] : lo;
    }
    const double top = hi + 1.0, no = nocc[blockIdx.x];
    if (tid < n && pd && pd[tid]) P[tid * pitch + tid] = top;
    __syncthreads();
    const double mu = block_sum(tid < n ? P[tid * pitch + tid] : 0.0, red) / n;
    const double l1 = no / (top - mu), l2 = (n - no) / (mu - lo), lam = (l2 < l1 ? l2 : l1) / n;
    for (int e = tid; e < n * n; e += blockDim.x) {
        const int i = e / n, j = e - i * n;
        const double x = P[i * pitch + j];
        P[i * pitch + j] = lam * ((i == j ? mu : 0.0) - x) + (i == j ? no / n : 0.0);
    }
    const int tiles = nt * (nt + 1) / 2;
    int fin = 0;
    for (int step = 0; step < maxit; ++step) {
        __syncthreads();   // P is complete
        for (int t = warp; t < tiles; t += kPurifyWarps) {
            int ti = 0, tj = t;
            while (tj > ti) tj -= ++ti;
            double acc[2][2][2];
            tile_product(P, P, pitch, np, 16 * ti, 16 * tj, lane, acc);
#pragma unroll
            for (int a = 0; a < 2; ++a)
#pragma unroll
                for (int b = 0; b < 2; ++b)
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        const int i = 16 * ti + 8 * a + (lane >> 2), j = 16 * tj + 8 * b + 2 * (lane & 3) + c;
                        if (j <= i) {
                            P2[i * pitch + j] = acc[a][b][c];
                            P2[j * pitch + i] = acc[a][b][c];
                        }
                    }
        }
        __syncthreads();
        // tr(P - P^2), tr(P^2 - P^3)
        double den = tid < n ? P[tid * pitch + tid] - P2[tid * pitch + tid] : 0.0;
        double num = tid < n ? P2[tid * pitch + tid] : 0.0;
        for (int i = warp; i < n; i += kPurifyWarps)
            for (int j = lane; j < n; j += 32) num = fma(-P2[i * pitch + j], P[i * pitch + j], num);
        den = block_sum(den, red);
        num = block_sum(num, red);
        fin = fabs(den) < tol * n;
        if (fin) break;   // uniform over the block
        double c = num / den;
        c = c < 0.0 ? 0.0 : (c > 1.0 ? 1.0 : c);
        const bool up = c >= 0.5;
        const double a0 = up ? 0.0 : (1.0 - 2.0 * c), a1 = 1.0 + c;
        const double inv = 1.0 / (up ? (c > 1e-300 ? c : 1e-300) : ((1.0 - c) > 1e-300 ? (1.0 - c) : 1e-300));
        double acc[kPurifyRounds][2][2][2];
#pragma unroll
        for (int r = 0; r < kPurifyRounds; ++r) {
            const int t = warp + r * kPurifyWarps;
            if (t < tiles) {
                int ti = 0, tj = t;
                while (tj > ti) tj -= ++ti;
                tile_product(P2, P, pitch, np, 16 * ti, 16 * tj, lane, acc[r]);
            }
        }
        __syncthreads();   // every warp has read P
#pragma unroll
        for (int r = 0; r < kPurifyRounds; ++r) {
            const int t = warp + r * kPurifyWarps;
            if (t < tiles) {
                int ti = 0, tj = t;
                while (tj > ti) tj -= ++ti;
#pragma unroll
                for (int a = 0; a < 2; ++a)
#pragma unroll
                    for (int b = 0; b < 2; ++b)
#pragma unroll
                        for (int k = 0; k < 2; ++k) {
                            const int i = 16 * ti + 8 * a + (lane >> 2), j = 16 * tj + 8 * b + 2 * (lane & 3) + k;
                            if (j <= i) {
                                const double x = fma(a0, P[i * pitch + j], fma(a1, P2[i * pitch + j], -acc[r][a][b][k])) * inv;
                                P[i * pitch + j] = x;
                                P[j * pitch + i] = x;
                            }
                        }
            }
        }
    }
    __syncthreads();
    double *o = Pout + (int64_t)blockIdx.x * n * n;
    for (int e = tid; e < n * n; e += blockDim.x) {
        const int i = e / n, j = e - i * n;
        o[e] = P[i * pitch + j];
    }
    if (tid == 0 && done) done[blockIdx.x] = fin;
}

// ---- x with A x = b for a batch of small systems, one warp each: Gauss-Jordan
// elimination with partial pivoting, lane j holding row j of [A | b] in
// registers (the first largest pivot on a tie; a singular system gives
// non-finite x).  The same elimination in tensor operations took about 100
// launches for the nine rows of a DIIS step: an iteration of 32 clusters in eight
// buckets 4.5 -> 2.9 ms.  C columns are compiled in.
template <int C>
__global__ void __launch_bounds__(128) solve_small_kernel(int nmat, int n, const double *__restrict__ A,
                                                          const double *__restrict__ b, double *__restrict__ x)
{
    const int m = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (m >= nmat) return;   // whole warps
    double row[C], rhs = lane < n ? b[(int64_t)m * n + lane] : 0.0;
#pragma unroll
    for (int j = 0; j < C; ++j) row[j] = lane < n && j < n ? A[((int64_t)m * n + lane) * n + j] : 0.0;
    int at = lane;   // the row of the permuted system that this lane holds
#pragma unroll
    for (int j = 0; j < C; ++j) {
        if (j < n) {   // uniform over the warp
            // the pivot among the rows not yet used: rows at >= j
            double best = lane < n && at >= j ? fabs(row[j]) : -1.0;
            if (!(best == best)) best = INFINITY;   // a NaN column is its own pivot
            double top = best;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const double y = __shfl_xor_sync(0xffffffffu, top, o);
                top = y > top ? y : top;
            }
            // (of several largest ones the one that comes first in row order)
            const unsigned first = __reduce_min_sync(0xffffffffu, best == top ? (unsigned)at : 64u);
            // rows first and j change places
            const bool is_pivot = at == (int)first && lane < n;
            if (is_pivot)
                at = j;
            else if (at == j)
                at = (int)first;
            const int src = __ffs((int)__ballot_sync(0xffffffffu, is_pivot)) - 1;
            const double inv = 1.0 / __shfl_sync(0xffffffffu, row[j], src);
            const double f = row[j], pr = __shfl_sync(0xffffffffu, rhs, src) * inv;
#pragma unroll
            for (int k = 0; k < C; ++k) {
                const double p = __shfl_sync(0xffffffffu, row[k], src) * inv;
                row[k] = is_pivot ? p : row[k] - f * p;
            }
            rhs = is_pivot ? pr : rhs - f * pr;
        }
    }
    if (lane < n) x[(int64_t)m * n + at] = rhs;
}

}  // namespace

extern "C" {

int pqb_solve_small(int nmat, int n, const double *A, const double *b, double *x, void *stream)
{
    if (nmat < 0 || n <= 0 || !A || !b || !x) return PQB_E_ARG;
    if (n > 17) return PQB_E_SHAPE;
    if (nmat == 0) return PQB_OK;
    const unsigned grid = (unsigned)(((int64_t)nmat + 3) / 4);
    cudaStream_t st = (cudaStream_t)stream;
    if (n <= 9)
        solve_small_kernel<9><<<grid, 128, 0, st>>>(nmat, n, A, b, x);
    else
        solve_small_kernel<17><<<grid, 128, 0, st>>>(nmat, n, A, b, x);
    return cudaGetLastError() == cudaSuccess ? PQB_OK : PQB_E_CUDA;
}

int pqb_purify(int nmat, int n, const double *F, const double *nocc, const unsigned char *pad, double *P, int *done,
               int maxit, double tol, void *stream)
{
    if (nmat < 0 || n <= 0 || maxit < 0 || !F || !nocc || !P) return PQB_E_ARG;
    if (n > kPurifyMax) return PQB_E_SHAPE;
    if (nmat == 0) return PQB_OK;
    const int np = (n + 15) / 16 * 16;
    const size_t bytes = sizeof(double) * 2 * np * (np + 4);
    if (cudaFuncSetAttribute(purify_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)(sizeof(double) * 2 * kPurifyMax * (kPurifyMax + 4))) != cudaSuccess)
        return PQB_E_CUDA;
    purify_kernel<<<nmat, kPurifyWarps * 32, bytes, (cudaStream_t)stream>>>(n, F, nocc, pad, P, done, maxit, tol);
    return cudaGetLastError() == cudaSuccess ? PQB_OK : PQB_E_CUDA;
}

int pqb_purify_step(int nmat, int n, const double *P, const double *P2, const double *P3, double *P_out, int *done,
                    double tol, void *stream)
{
    if (nmat < 0 || n <= 0 || !P || !P2 || !P3 || !P_out) return PQB_E_ARG;
    if (nmat == 0) return PQB_OK;
    purify_step_kernel<<<nmat, kPurifyThreads, 0, (cudaStream_t)stream>>>(n, P, P2, P3, P_out, done, tol);
    return cudaGetLastError() == cudaSuccess ? PQB_OK : PQB_E_CUDA;
}

}  // extern "C"
