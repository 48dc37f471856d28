// Numerical-integration kernels of the DFT path (the reference's MG2 grid,
// PyQuante/MG2.py:50-250, with Becke's partitioning of
// PyQuante/MolecularGrid.py:228-263, and the SVWN functional of
// PyQuante/DFunctionals.py:76-138,319-389,603-623):
//   * becke_weights_kernel: the cell weight of every grid point
//     w = w_atomic P_owner / sum_j P_j, P_j = prod_{k != j} s(mu'_jk),
//     mu_jk = (|r - R_j| - |r - R_k|)/|R_j - R_k|, mu' = mu + a_jk (1 - mu^2),
//     s = (1 - f3(mu'))/2 with f3 three applications of 1.5 x - 0.5 x^3;
//   * grid_amps_kernel: basis amplitudes B[g][i] = N_i x^l y^m z^n
//     sum_p c_p exp(-alpha_p r^2) (CGBF.amp, PyQuante/CGBF.py:116-120) --
//     the HBM-bound write of the grid path;
//   * grid_density_kernel: rho_g = sum_ij B_gi D_ij B_gj (MG2.bdb), and
//     grid_fock_kernel: F_ij = sum_g B_gi v_g B_gj (the Fxc assembly of
//     PyQuante/dft.py:29-65), both on FP64 tensor-core tiles over the
//     triangle of their symmetric matrix;
//   * grid_rowdot_kernel: out_g = sum_i A_gi B_gi;
//   * xc_svwn_kernel: Slater exchange (X-alpha 2/3, per spin) plus VWN
//     correlation per point, weighted: w f_xc, w v_a, w v_b.
#include <cmath>
#include <cstdint>

#include <cuda_runtime.h>

#include "../../include/pyquante_b200.h"
#include "dmma.cuh"

using namespace pqb;

namespace {

__global__ void becke_weights_kernel(int npts, const double *__restrict__ pts, const int *__restrict__ owner, int nat,
                                     const double *__restrict__ atoms, const double *__restrict__ adj,
                                     double *__restrict__ w)
{
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < npts; g += gridDim.x * blockDim.x) {
        const double px = pts[4 * g], py = pts[4 * g + 1], pz = pts[4 * g + 2];
        double sum = 0.0, own = 0.0;
        const int o = owner[g];
        for (int j = 0; j < nat; ++j) {
            const double xj = atoms[3 * j], yj = atoms[3 * j + 1], zj = atoms[3 * j + 2];
            const double rjp = sqrt((px - xj) * (px - xj) + (py - yj) * (py - yj) + (pz - zj) * (pz - zj));
            double P = 1.0;
            for (int k = 0; k < nat && P != 0.0; ++k) {
                if (k == j) continue;
                const double xk = atoms[3 * k], yk = atoms[3 * k + 1], zk = atoms[3 * k + 2];
                const double rkp = sqrt((px - xk) * (px - xk) + (py - yk) * (py - yk) + (pz - zk) * (pz - zk));
                const double rjk = sqrt((xj - xk) * (xj - xk) + (yj - yk) * (yj - yk) + (zj - zk) * (zj - zk));
                double mu = (rjp - rkp) / rjk;
                mu += adj[j * nat + k] * (1.0 - mu * mu);
#pragma unroll
                for (int it = 0; it < 3; ++it) mu = 1.5 * mu - 0.5 * mu * mu * mu;
                P *= 0.5 * (1.0 - mu);
            }
            sum += P;
            if (j == o) own = P;
        }
        w[g] = sum > 0.0 ? pts[4 * g + 3] * own / sum : 0.0;
    }
}

__global__ void grid_amps_kernel(int n, const double *__restrict__ origin, const int *__restrict__ powers,
                                 const int *__restrict__ prim_off, const double *__restrict__ exps,
                                 const double *__restrict__ cn, const double *__restrict__ norms, int npts,
                                 const double *__restrict__ pts, double *__restrict__ B)
{
    const int64_t total = (int64_t)npts * n;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        const int g = (int)(t / n), i = (int)(t - (int64_t)g * n);
        const double dx = pts[4 * g] - origin[3 * i], dy = pts[4 * g + 1] - origin[3 * i + 1],
                     dz = pts[4 * g + 2] - origin[3 * i + 2];
        const double r2 = dx * dx + dy * dy + dz * dz;
        double poly = 1.0;
        for (int k = 0; k < powers[3 * i]; ++k) poly *= dx;
        for (int k = 0; k < powers[3 * i + 1]; ++k) poly *= dy;
        for (int k = 0; k < powers[3 * i + 2]; ++k) poly *= dz;
        double s = 0.0;
        for (int p = prim_off[i]; p < prim_off[i + 1]; ++p) s += cn[p] * exp(-exps[p] * r2);
        B[t] = norms[i] * poly * s;
    }
}

// one warp per row g: out[g] = sum_i A[g][i] B[g][i]
__global__ void grid_rowdot_kernel(int npts, int n, const double *__restrict__ A, const double *__restrict__ B,
                                   double *__restrict__ out)
{
    const int lane = threadIdx.x & 31;
    for (int g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; g < npts; g += (gridDim.x * blockDim.x) >> 5) {
        const double *a = A + (int64_t)g * n, *b = B + (int64_t)g * n;
        double s = 0.0;
        for (int i = lane; i < n; i += 32) s = fma(__ldg(a + i), __ldg(b + i), s);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (lane == 0) out[g] = s;
    }
}

// ---- density: rho_g = sum_ij B_gi D_ij B_gj as FP64 tensor-core tiles.
// With W_kj = D_kj + D_jk below the diagonal and D_kk on it, rho_g =
// sum_j B_gj sum_(k >= j) B_gk W_kj: half the products of B D.  A block takes
// 128 points and walks the 32-column strips j of W with k from the strip's
// start on; the strip's products are dotted with B_gj in registers, so B D is
// never written.  The strip's width (32, 40 or 48) is the one that pads the
// triangle least: 32 at N = 200.  Bound by the FP64 tensor rate (72 % of the
// pipe): (H2O)8 / 6-31G** (148,992 points, N = 200) takes 0.29 ms (20.5 TFLOP/s of
// the triangle's operations); the full DGEMM and the row dot took 0.46 + 0.08 ms.
constexpr int kDensRows = 128, kDensK = 16, kDensStages = 3, kDensPitchA = kDensK + 4;

template <int NF> struct DensLayout {
    static constexpr int cols = 8 * NF;
    static constexpr int pitchB = (cols + 15) / 16 * 16 + 4;   // 4 mod 16: fragment reads hit distinct banks
    static constexpr int stage = kDensRows * kDensPitchA + kDensK * pitchB;
    static constexpr size_t bytes = sizeof(double) * kDensStages * stage;
};

// products a point of the strips of 8 nf columns
int64_t dens_cost(int n, int nf)
{
    const int c = 8 * nf;
    int64_t s = 0;
    for (int j0 = 0; j0 < n; j0 += c) s += (int64_t)c * ((n + kDensK - 1) / kDensK * kDensK - j0 / kDensK * kDensK);
    return s;
}

int dens_nf(int n)
{
    int nf = 6;   // (the wider strip on a tie: fewer passes over B)
    for (int t = 5; t >= 4; --t)
        if (dens_cost(n, t) < dens_cost(n, nf)) nf = t;
    return nf;
}

int dens_rows(int n) { return (n + kDensK - 1) / kDensK * kDensK; }
int dens_cols(int n)
{
    const int c = 8 * dens_nf(n);
    return (n + c - 1) / c * c;
}

// W, zero-padded to nr rows and np columns
__global__ void fold_density_kernel(int n, int nr, int np, const double *__restrict__ D, double *__restrict__ W)
{
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < nr * np; t += gridDim.x * blockDim.x) {
        const int k = t / np, j = t - k * np;
        double w = 0.0;
        if (k < n && j <= k) w = k == j ? D[(int64_t)k * n + k] : D[(int64_t)k * n + j] + D[(int64_t)j * n + k];
        W[t] = w;
    }
}

// VEC: B starts on a 16-byte boundary, and its rows are copied 16 bytes at a
// time; with n odd every second row starts 8 bytes past one, and its copies
// start one element early (a row's shared image is shifted by sh = 0 or 1).
template <int NF, bool VEC>
__global__ void __launch_bounds__(128) grid_density_kernel(int npts, int n, int np, const double *__restrict__ B,
                                                           const double *__restrict__ W, double *__restrict__ rho,
                                                           int stride, int copies)
{
    using Lay = DensLayout<NF>;
    extern __shared__ __align__(16) double sm[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t g0 = (int64_t)blockIdx.x * kDensRows;
    const int nk = (n + kDensK - 1) / kDensK, njt = np / Lay::cols;
    // what this thread copies in every step: eight 16-byte pieces of A (rows tid/8
    // + 16 i, one parity, hence one shift), with n odd also the ninth piece of row
    // tid, and up to NPW pieces of W
    constexpr int NPW = (kDensK * Lay::cols / 2 + 127) / 128;
    const int ra = tid >> 3, qa = 2 * (tid & 7);
    const int sha = VEC ? (int)(((g0 + ra) * n) & 1) : 0, sh9 = (int)(((g0 + tid) * n) & 1);
    const double *Ag = B + (g0 + ra) * n - sha + qa, *A9 = B + (g0 + tid) * n + kDensK - 1;
    const int rows = npts - g0 < kDensRows ? (int)(npts - g0) : kDensRows;
    int woff[NPW], wsm[NPW];
#pragma unroll
    for (int i = 0; i < NPW; ++i) {
        const int e = tid + 128 * i, k = e / (Lay::cols / 2), j = 2 * (e % (Lay::cols / 2));
        woff[i] = k * np + j;
        wsm[i] = e < kDensK * Lay::cols / 2 ? kDensRows * kDensPitchA + k * Lay::pitchB + j : -1;
    }
    auto load = [&](int j0, int k0, int slot) {
        double *s = sm + slot * Lay::stage;
        if (VEC) {
            const int left = n - k0 + sha - qa, count = left > 1 ? 2 : (left > 0 ? left : 0);
            double *d = s + ra * kDensPitchA + qa;
            const double *a = Ag + k0;
#pragma unroll
            for (int i = 0; i < 8; ++i, a += (int64_t)16 * n, d += 16 * kDensPitchA) {
                const int c = ra + 16 * i < rows ? count : 0;
                cp_async16(d, c ? a : B, c);
            }
            if (n & 1) {
                const int c = tid < rows && sh9 && k0 + kDensK <= n ? 1 : 0;
                cp_async16(s + tid * kDensPitchA + kDensK, c ? A9 + k0 : B, c);
            }
        } else {
#pragma unroll
            for (int e = tid; e < kDensRows * kDensK; e += 128) {
                const int r = e / kDensK, k = e % kDensK;
                const bool ok = r < rows && k0 + k < n;
                cp_async8(s + r * kDensPitchA + k, ok ? B + (g0 + r) * n + k0 + k : B, ok);
            }
        }
        const double *w = W + (int64_t)k0 * np + j0;
#pragma unroll
        for (int i = 0; i < NPW; ++i)
            if (wsm[i] >= 0) cp_async16(s + wsm[i], w + woff[i], 2);
    };
    // the shift of this thread's rows (warp 32 + 8 m + lane / 4: one parity)
    const int sh = VEC ? (int)(((g0 + (lane >> 2)) * n) & 1) : 0;
    // the sequence of (strip, k block) steps, walked twice: by the loads and, two
    // steps behind, by the products
    int lj = 0, lk = 0, step = 0;
    auto issue = [&]() {
        if (lj < njt) {
            load(lj * Lay::cols, lk * kDensK, step % kDensStages);
            if (++lk >= nk) {
                ++lj;
                lk = lj * Lay::cols / kDensK;
            }
        }
        ++step;
        cp_async_commit();
    };
#pragma unroll
    for (int s = 0; s < kDensStages - 1; ++s) issue();
    double rs[4] = {0.0, 0.0, 0.0, 0.0};
    int slot = 0;
    for (int jt = 0; jt < njt; ++jt) {
        double acc[4][NF][2];
#pragma unroll
        for (int m = 0; m < 4; ++m)
#pragma unroll
            for (int c = 0; c < NF; ++c) acc[m][c][0] = acc[m][c][1] = 0.0;
        for (int kt = jt * Lay::cols / kDensK; kt < nk; ++kt) {
            cp_async_wait<kDensStages - 2>();
            __syncthreads();   // this step has landed; the readers of the step before are done
            issue();
            const double *As = sm + slot * Lay::stage + (warp * 32 + (lane >> 2)) * kDensPitchA + (lane & 3) + sh;
            const double *Bs = sm + slot * Lay::stage + kDensRows * kDensPitchA + (lane & 3) * Lay::pitchB + (lane >> 2);
            slot = slot + 1 == kDensStages ? 0 : slot + 1;
#pragma unroll
            for (int k = 0; k < kDensK; k += 4) {
                double a[4], b[NF];
#pragma unroll
                for (int m = 0; m < 4; ++m) a[m] = As[8 * m * kDensPitchA + k];
#pragma unroll
                for (int c = 0; c < NF; ++c) b[c] = Bs[k * Lay::pitchB + 8 * c];
#pragma unroll
                for (int m = 0; m < 4; ++m)
#pragma unroll
                    for (int c = 0; c < NF; ++c) dmma(acc[m][c], a[m], b[c]);
            }
        }
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const int64_t g = g0 + warp * 32 + 8 * m + (lane >> 2);
#pragma unroll
            for (int c = 0; c < NF; ++c) {
                const int j = jt * Lay::cols + 8 * c + 2 * (lane & 3);
                if (g < npts && j < n) rs[m] = fma(acc[m][c][0], __ldg(B + g * n + j), rs[m]);
                if (g < npts && j + 1 < n) rs[m] = fma(acc[m][c][1], __ldg(B + g * n + j + 1), rs[m]);
            }
        }
    }
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        double s = rs[m];
        s += __shfl_xor_sync(0xffffffffu, s, 1);
        s += __shfl_xor_sync(0xffffffffu, s, 2);
        const int64_t g = g0 + warp * 32 + 8 * m + (lane >> 2);
        if ((lane & 3) == 0 && g < npts)
            for (int c = 0; c < copies; ++c) rho[g * stride + c] = s;
    }
}

template <int NF>
cudaError_t launch_density(int npts, int n, int np, const double *B, const double *W, double *rho, int stride, int copies,
                           cudaStream_t st)
{
    using Lay = DensLayout<NF>;
    const bool vec = (reinterpret_cast<uintptr_t>(B) & 15) == 0;
    auto kern = vec ? grid_density_kernel<NF, true> : grid_density_kernel<NF, false>;
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Lay::bytes);
    if (e != cudaSuccess) return e;
    kern<<<(unsigned)(((int64_t)npts + kDensRows - 1) / kDensRows), 128, Lay::bytes, st>>>(npts, n, np, B, W, rho, stride,
                                                                                             copies);
    return cudaGetLastError();
}

// ---- F_ij = sum_g B_gi v_g B_gj as FP64 tensor-core tiles of the lower
// triangle.  The columns form strips of T = 8 TF; a block takes a range of
// points and a group of strip pairs, one T x T tile a warp, so that each 16
// points' rows of B go through shared memory once for all the group's tiles
// (v multiplied into one factor's fragments; rows copied and shifted as above).  The ranges' partial tiles are
// added in a fixed order.  Same bound: 0.28 ms at the size above; the full
// DGEMM took 0.59 ms and the pass that wrote v B 0.10 ms; one block per strip
// pair, which reads B once per pair, 0.64 ms.
constexpr int kFockK = 16, kFockStages = 3;

template <int TF> struct FockLayout {
    // tiles of a group: five strips' triangle at most, or (TF = 4) four strips against four
    static constexpr int warps = TF == 4 ? 16 : 15;
};

__host__ __device__ constexpr int fock_pitch(int cols) { return (cols + 15) / 16 * 16 + 4; }

template <int TF, bool VEC>
__global__ void __launch_bounds__(FockLayout<TF>::warps * 32, 1)
grid_fock_kernel(int npts, int n, const double *__restrict__ B, const double *__restrict__ v, int nt, int macro,
                 int chunk, double *__restrict__ part)
{
    constexpr int T = 8 * TF;
    extern __shared__ __align__(16) double sm[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    // group (I >= J): strips [I macro, ..) against strips [J macro, ..)
    int I = 0, J = blockIdx.x;
    while (J > I) J -= ++I;
    const int si0 = I * macro, si = min(macro, nt - si0), sj0 = J * macro, sj = I == J ? 0 : min(macro, nt - sj0);
    const int ci = si * T, cols = ci + sj * T, pitch = fock_pitch(cols + (VEC ? 4 : 0)), stage = kFockK * pitch + kFockK;
    // this warp's tile: strips a, b of the shared rows
    int a = 0, b = warp;
    bool active;
    if (I == J) {
        while (b > a) b -= ++a;
        active = a < si;
    } else {
        a = warp / macro;
        b = warp % macro;
        active = a < si && b < sj;
        b += si;
    }
    const int64_t gb = (int64_t)blockIdx.y * chunk, ge = gb + chunk < npts ? gb + chunk : npts;
    const int steps = ge > gb ? (int)((ge - gb + kFockK - 1) / kFockK) : 0;
    auto load = [&](int t, int slot) {
        double *s = sm + slot * stage;
        const int64_t gs = gb + (int64_t)t * kFockK;
        for (int k = warp; k < kFockK; k += nw) {
            const double *row = B + (gs + k) * n;
            if (VEC) {
                // each run of columns (the I strips, the J strips) from the 16-byte boundary at or before it
                const int sh = (int)(((gs + k) * n) & 1);
                for (int run = 0; run < (I == J ? 1 : 2); ++run) {
                    const int c0 = run ? sj0 * T : si0 * T, len = (run ? cols - ci : ci) + sh;
                    double *d = s + k * pitch + (run ? ci + 2 : 0);
                    for (int c = 2 * lane; c < len; c += 64) {
                        const int left = n - c0 + sh - c;
                        const int count = gs + k < ge ? (left > 1 ? 2 : (left > 0 ? left : 0)) : 0;
                        cp_async16(d + c, count ? row + c0 - sh + c : B, count);
                    }
                }
                continue;
            }
            for (int c = lane; c < cols; c += 32) {
                const int col = c < ci ? si0 * T + c : sj0 * T + c - ci;
                const bool ok = gs + k < ge && col < n;
                cp_async8(s + k * pitch + c, ok ? row + col : B, ok);
            }
        }
        if (threadIdx.x < kFockK) {
            const int64_t g = gs + threadIdx.x;
            cp_async8(s + kFockK * pitch + threadIdx.x, g < ge ? v + g : v, g < ge);
        }
    };
    double acc[TF][TF][2];
#pragma unroll
    for (int m = 0; m < TF; ++m)
#pragma unroll
        for (int c = 0; c < TF; ++c) acc[m][c][0] = acc[m][c][1] = 0.0;
#pragma unroll
    for (int s = 0; s < kFockStages - 1; ++s) {
        if (s < steps) load(s, s);
        cp_async_commit();
    }
    int slot = 0, next = kFockStages - 1;
    for (int t = 0; t < steps; ++t) {
        cp_async_wait<kFockStages - 2>();
        __syncthreads();   // stage t has landed; the readers of the stage that is loaded next are done
        if (t + kFockStages - 1 < steps) load(t + kFockStages - 1, next);
        cp_async_commit();
        const double *s = sm + slot * stage;
        next = slot;
        slot = slot + 1 == kFockStages ? 0 : slot + 1;
        if (active) {
            // (the J strips of an off-diagonal group start two elements further on)
            const int sh = VEC ? (int)(((gb + (lane & 3)) * n) & 1) : 0;
            const double *As = s + (lane & 3) * pitch + a * T + (lane >> 2) + sh,
                         *Bs = As + (b - a) * T + (VEC && I != J ? 2 : 0);
#pragma unroll
            for (int k = 0; k < kFockK; k += 4) {
                const double w = s[kFockK * pitch + k + (lane & 3)];
                double x[TF], y[TF];
#pragma unroll
                for (int m = 0; m < TF; ++m) x[m] = w * As[k * pitch + 8 * m];
#pragma unroll
                for (int c = 0; c < TF; ++c) y[c] = Bs[k * pitch + 8 * c];
#pragma unroll
                for (int m = 0; m < TF; ++m)
#pragma unroll
                    for (int c = 0; c < TF; ++c) dmma(acc[m][c], x[m], y[c]);
            }
        }
    }
    if (active) {
        const int it = si0 + a, jt = I == J ? sj0 + b : sj0 + b - si;
        double *o = part + ((int64_t)blockIdx.y * (nt * (nt + 1) / 2) + it * (it + 1) / 2 + jt) * T * T;
#pragma unroll
        for (int m = 0; m < TF; ++m)
#pragma unroll
            for (int c = 0; c < TF; ++c) {
                const int e = (8 * m + (lane >> 2)) * T + 8 * c + 2 * (lane & 3);
                o[e] = acc[m][c][0];
                o[e + 1] = acc[m][c][1];
            }
    }
}

// F[i][j] = F[j][i] = the sum of the point ranges' partial tiles: eight
// threads an element, each every eighth range.
__global__ void __launch_bounds__(256) grid_fock_sum_kernel(int n, int T, int npair, int splits,
                                                            const double *__restrict__ part, double *__restrict__ F)
{
    __shared__ double red[8][33];
    int it = 0, p = blockIdx.x;
    while (p > it) p -= ++it;
    const int x = threadIdx.x & 31, y = threadIdx.x >> 5, e = blockIdx.y * 32 + x;
    const bool in = e < T * T;
    double s = 0.0;
    if (in)
        for (int k = y; k < splits; k += 8) s += part[((int64_t)k * npair + blockIdx.x) * T * T + e];
    red[y][x] = s;
    __syncthreads();
    if (y == 0 && in) {
        const int i = it * T + e / T, j = p * T + e % T;
        if (i < n && j <= i) {
#pragma unroll
            for (int k = 1; k < 8; ++k) s += red[k][x];
            F[(int64_t)i * n + j] = s;
            F[(int64_t)j * n + i] = s;
        }
    }
}

// Up to five strips (one group) of the width that pads the triangle least
// (N = 200: five of 40, 24,000 products a point against the square's 40,000);
// more functions go in strips of 32, grouped four by four.  The points are
// split into as many ranges as fill the GPU once (six times with several
// groups, whose blocks differ), 64 points at least.
struct FockSplit {
    int tf, nt, npair, macro, groups, warps, splits, chunk;
};

FockSplit fock_split(int npts, int n)
{
    FockSplit f{};
    int64_t best = 0;
    for (int tf = 1; tf <= 5; ++tf) {
        const int nt = (n + 8 * tf - 1) / (8 * tf);
        if (nt > 5) continue;
        // products, and the fragments read for them
        const int64_t cost = (int64_t)nt * (nt + 1) / 2 * tf * (tf * 4 + 4);
        if (!f.tf || cost < best) {
            best = cost;
            f.tf = tf;
        }
    }
    f.macro = 5;
    if (!f.tf) {
        f.tf = 4;
        f.macro = 4;
    }
    f.nt = (n + 8 * f.tf - 1) / (8 * f.tf);
    f.npair = f.nt * (f.nt + 1) / 2;
    const int mt = (f.nt + f.macro - 1) / f.macro;
    f.groups = mt * (mt + 1) / 2;
    f.warps = mt > 1 ? 16 : f.npair;
    // one block an SM where a block is that large (one wave), else 32 warps an SM
    int64_t s = f.warps > 8 ? (f.groups == 1 ? 148 : 148 * 6 / f.groups) : 148 * 32 / f.warps;
    const int64_t most = (npts + 63) / 64;
    if (s > most) s = most;
    if (s < 1) s = 1;
    f.chunk = (int)(((npts + s - 1) / s + kFockK - 1) / kFockK * kFockK);
    if (f.chunk < kFockK) f.chunk = kFockK;
    f.splits = (npts + f.chunk - 1) / f.chunk;
    if (f.splits < 1) f.splits = 1;
    return f;
}

template <int TF>
cudaError_t launch_fock(const FockSplit &f, int npts, int n, const double *B, const double *v, double *part,
                        cudaStream_t st)
{
    const bool vec = (reinterpret_cast<uintptr_t>(B) & 15) == 0;
    auto kern = vec ? grid_fock_kernel<TF, true> : grid_fock_kernel<TF, false>;
    const int strips = f.groups > 1 ? 2 * f.macro : f.nt;
    const size_t bytes = sizeof(double) * kFockStages * (kFockK * fock_pitch(strips * 8 * TF + 4) + kFockK);
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    if (e != cudaSuccess) return e;
    kern<<<dim3(f.groups, f.splits), f.warps * 32, bytes, st>>>(npts, n, B, v, f.nt, f.macro, f.chunk, part);
    return cudaGetLastError();
}

__device__ __forceinline__ double vwn_xx(double x, double b, double c) { return x * x + b * x + c; }

__device__ double vwn_eps(double x, double a, double x0, double b, double c)
{
    const double q = sqrt(4.0 * c - b * b);
    return a * (log(x * x / vwn_xx(x, b, c)) - b * (x0 / vwn_xx(x0, b, c)) * log((x - x0) * (x - x0) / vwn_xx(x, b, c)) +
                (2.0 * b / q) * (1.0 - (x0 * (2.0 * x0 + b) / vwn_xx(x0, b, c))) * atan(q / (2.0 * x + b)));
}

__device__ double vwn_deps(double x, double a, double x0, double b, double c)
{
    const double q = sqrt(4.0 * c - b * b), t = 2.0 * x + b;
    return a * (2.0 / x - t / vwn_xx(x, b, c) - 4.0 * b / (t * t + q * q) -
                (b * x0 / vwn_xx(x0, b, c)) * (2.0 / (x - x0) - t / vwn_xx(x, b, c) - 4.0 * (2.0 * x0 + b) / (t * t + q * q)));
}

// VWN parameters (A, x0, b, c) of the paramagnetic and ferromagnetic fits
// (Vosko, Wilk and Nusair, Can. J. Phys. 58, 1200 (1980)), as the reference uses them
#define VWN_P 0.0310907, -0.10498, 3.72744, 12.9352
#define VWN_F 0.01554535, -0.32500, 7.06042, 13.0045

__global__ void xc_svwn_kernel(int npts, const double *__restrict__ rhoa, const double *__restrict__ rhob,
                               const double *__restrict__ w, double *__restrict__ wf, double *__restrict__ wva,
                               double *__restrict__ wvb)
{
    const double tol = 1e-10;
    const double fac = -2.25 * (2.0 / 3.0) * cbrt(3.0 / (4.0 * M_PI));
    for (int g = blockIdx.x * blockDim.x + threadIdx.x; g < npts; g += gridDim.x * blockDim.x) {
        const double na = rhoa[g], nb = rhob[g];
        double f = 0.0, va = 0.0, vb = 0.0;
        // Slater exchange, per spin
        {
            const double ra = na < tol ? 0.0 : na, rb = nb < tol ? 0.0 : nb;
            const double a3 = cbrt(ra), b3 = cbrt(rb);
            f = fac * (ra * a3 + rb * b3);
            va = (4.0 / 3.0) * fac * a3;
            vb = (4.0 / 3.0) * fac * b3;
        }
        // VWN correlation
        const double rho = na + nb;
        if (rho >= tol) {
            const double zeta = (na - nb) / rho;
            const double x = pow(3.0 / (4.0 * M_PI) / rho, 1.0 / 6.0);
            const double ep = vwn_eps(x, VWN_P), dep = vwn_deps(x, VWN_P);
            const double gz = 1.125 * (pow(1.0 + zeta, 4.0 / 3.0) + pow(1.0 - zeta, 4.0 / 3.0) - 2.0);
            if (gz < tol) {
                f += ep * rho;
                va += ep - (x / 6.0) * dep;
                vb += ep - (x / 6.0) * dep;
            } else {
                const double ef = vwn_eps(x, VWN_F), def = vwn_deps(x, VWN_F);
                const double e = ep + gz * (ef - ep);
                const double dg = 1.5 * (cbrt(1.0 + zeta) - cbrt(1.0 - zeta));
                const double dx = dep + gz * (def - dep), dgg = (ef - ep) * dg;
                f += e * rho;
                va += e - (x / 6.0) * dx + dgg * (1.0 - zeta);
                vb += e - (x / 6.0) * dx - dgg * (1.0 + zeta);
            }
        }
        wf[g] = w[g] * f;
        wva[g] = w[g] * va;
        wvb[g] = w[g] * vb;
    }
}

int grid_of(int64_t total, int per)
{
    const int64_t g = (total + per - 1) / per;
    return (int)(g < 148 * 32 ? (g > 0 ? g : 1) : 148 * 32);
}

}  // namespace

extern "C" {

int pqb_becke_weights(int npts, const double *pts, const int *owner, int natoms, const double *atom_xyz,
                      const double *adjust, double *w, void *stream)
{
    if (npts < 0 || natoms <= 0 || !pts || !owner || !atom_xyz || !adjust || !w) return PQB_E_ARG;
    if (npts == 0) return PQB_OK;
    becke_weights_kernel<<<grid_of(npts, 128), 128, 0, (cudaStream_t)stream>>>(npts, pts, owner, natoms, atom_xyz,
                                                                             adjust, w);
    return cudaGetLastError() == cudaSuccess ? PQB_OK : PQB_E_CUDA;
}

int pqb_grid_amps(int n, const double *origin, const int *powers, const int *prim_off, const double *exps,
                  const double *cn, const double *norms, int npts, const double *pts, double *B, void *stream)
{
    if (n <= 0 || npts < 0 || !origin || !powers || !prim_off || !exps || !cn || !norms || !pts || !B)
        return PQB_E_ARG;
    if (npts == 0) return PQB_OK;
    grid_amps_kernel<<<grid_of((int64_t)npts * n, 256), 256, 0, (cudaStream_t)stream>>>(n, origin, powers, prim_off,
                                                                                         exps, cn, norms, npts, pts, B);
    return cudaGetLastError() == cudaSuccess ? PQB_OK : PQB_E_CUDA;
}

int pqb_grid_rowdot(int npts, int n, const double *A, const double *B, double *out, void *stream)
{
    if (npts < 0 || n <= 0 || !A || !B || !out) return PQB_E_ARG;
    if (npts == 0) return PQB_OK;
    grid_rowdot_kernel<<<grid_of((int64_t)npts * 32, 256), 256, 0, (cudaStream_t)stream>>>(npts, n, A, B, out);
    return cudaGetLastError() == cudaSuccess ? PQB_OK : PQB_E_CUDA;
}

int64_t pqb_grid_work(int npts, int n)
{
    if (npts < 0 || n <= 0) return 0;
    const FockSplit f = fock_split(npts, n);
    const int64_t fock = (int64_t)f.splits * f.npair * 64 * f.tf * f.tf, dens = (int64_t)dens_rows(n) * dens_cols(n);
    return fock > dens ? fock : dens;
}

int pqb_grid_density(int npts, int n, const double *B, const double *D, double *rho, int stride, int copies,
                     double *work, void *stream)
{
    if (npts < 0 || n <= 0 || !B || !D || !rho || !work || copies < 1 || stride < copies ||
        (reinterpret_cast<uintptr_t>(work) & 15))
        return PQB_E_ARG;
    if (npts == 0) return PQB_OK;
    cudaStream_t st = (cudaStream_t)stream;
    const int nr = dens_rows(n), np = dens_cols(n);
    fold_density_kernel<<<grid_of((int64_t)nr * np, 256), 256, 0, st>>>(n, nr, np, D, work);
    cudaError_t e = cudaErrorInvalidValue;
    switch (dens_nf(n)) {
    case 4: e = launch_density<4>(npts, n, np, B, work, rho, stride, copies, st); break;
    case 5: e = launch_density<5>(npts, n, np, B, work, rho, stride, copies, st); break;
    case 6: e = launch_density<6>(npts, n, np, B, work, rho, stride, copies, st); break;
    }
    return e == cudaSuccess ? PQB_OK : PQB_E_CUDA;
}

int pqb_grid_fock(int npts, int n, const double *B, const double *v, double *F, double *work, void *stream)
{
    if (npts < 0 || n <= 0 || !B || !v || !F || !work) return PQB_E_ARG;
    cudaStream_t st = (cudaStream_t)stream;
    if (npts == 0) return cudaMemsetAsync(F, 0, sizeof(double) * n * n, st) == cudaSuccess ? PQB_OK : PQB_E_CUDA;
    const FockSplit f = fock_split(npts, n);
    cudaError_t e = cudaErrorInvalidValue;
    switch (f.tf) {
    case 1: e = launch_fock<1>(f, npts, n, B, v, work, st); break;
    case 2: e = launch_fock<2>(f, npts, n, B, v, work, st); break;
    case 3: e = launch_fock<3>(f, npts, n, B, v, work, st); break;
    case 4: e = launch_fock<4>(f, npts, n, B, v, work, st); break;
    case 5: e = launch_fock<5>(f, npts, n, B, v, work, st); break;
    }
    if (e != cudaSuccess) return PQB_E_CUDA;
    const int T = 8 * f.tf;
    grid_fock_sum_kernel<<<dim3(f.npair, (T * T + 31) / 32), 256, 0, st>>>(n, T, f.npair, f.splits, work, F);
    return cudaGetLastError() == cudaSuccess ? PQB_OK : PQB_E_CUDA;
}

int pqb_xc_svwn(int npts, const double *rhoa, const double *rhob, const double *w, double *wf, double *wva,
                double *wvb, void *stream)
{
    if (npts < 0 || !rhoa || !rhob || !w || !wf || !wva || !wvb) return PQB_E_ARG;
    if (npts == 0) return PQB_OK;
    xc_svwn_kernel<<<grid_of(npts, 128), 128, 0, (cudaStream_t)stream>>>(npts, rhoa, rhob, w, wf, wva, wvb);
    return cudaGetLastError() == cudaSuccess ? PQB_OK : PQB_E_CUDA;
}

}  // extern "C"
