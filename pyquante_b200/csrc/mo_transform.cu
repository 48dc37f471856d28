// AO -> MO integral transformation for the MP2 energy (the work of the
// reference's PyQuante/MP.py:20-75 TransformIntsMP2 and :77-97 MP2), on
// the packed integrals of pqb_eri_packed.
//
// The four quarter transformations are dense FP64 contractions; those over an
// index of a packed pair are kernels here, the two others cuBLAS DGEMMs from the
// host side:
//   * mo_contract_rows_kernel: the contraction over one index of (kl) of the
//     8-fold packed order (Src/cints.c:413-425);
//   * mo_unpack_rows_kernel: a batch of packed bra rows (ij| into dense
//     N x N matrices (ij|kl), for every kl, for callers with GEMMs of their own;
//   * mo_contract_pairs_kernel: the contraction over one index of the packed
//     AO pair of the half-transformed integrals, as FP64 tensor-core tiles
//     that gather the pair rows;
//   * mo_unpack_pairs_kernel: rows stored per packed AO pair into dense
//     (mu, nu) rows, symmetric;
//   * mo_pack_kernel: (ai|bj) into the reference's packed MO array at
//     ijkl2intindex(a, i, b, j);
//   * mp2_pairs_kernel: the pair energies
//       E_ab = sum_rs (ar|bs) (2 (ar|bs) - (as|br)) / (e_a + e_b - e_r - e_s).
#include <cstdint>

#include <cuda_runtime.h>

#include "../../include/pyquante_b200.h"
#include "dmma.cuh"

using namespace pqb;

namespace {

__device__ __forceinline__ int64_t pair_of(int64_t i, int64_t j)
{
    return i >= j ? i * (i + 1) / 2 + j : j * (j + 1) / 2 + i;
}

__device__ __forceinline__ int64_t packed_of(int64_t ij, int64_t kl)
{
    return ij >= kl ? ij * (ij + 1) / 2 + kl : kl * (kl + 1) / 2 + ij;
}

// out[r][k][l] = (IJ_r|kl), IJ_r = row0 + r.  A block takes a 32 x 32 tile
// k >= l of four consecutive bra rows: each packed element is read once, along
// l where the row holds it (kl <= IJ) and four neighbours IJ at a time, one
// 32-byte sector, where a later row does, and goes out twice, the transposed
// half through shared memory.  Bound by the 8 N^2 bytes a row that it writes:
// all 11,325 rows at N = 150 (2.04 GB out) take 0.95 ms, 1.65 ms
// with one thread per output element (64-bit divisions, strided reads of every
// element twice).
constexpr int kUnpackRows = 4;

__global__ void __launch_bounds__(256) mo_unpack_rows_kernel(const double *__restrict__ ints, int nbf, int64_t row0,
                                                             int nrows, int ntile2, double *__restrict__ out)
{
    __shared__ double s[kUnpackRows][32][33];
    const int lane = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int tile = blockIdx.x % ntile2, r0 = (int)(blockIdx.x / ntile2) * kUnpackRows;
    int kt = (int)((sqrtf(8.0f * tile + 1.0f) - 1.0f) * 0.5f);
    while (kt * (kt + 1) / 2 > tile) --kt;
    while ((kt + 1) * (kt + 2) / 2 <= tile) ++kt;
    const int lt = tile - kt * (kt + 1) / 2;
    const int64_t IJ0 = row0 + r0;
    const int rows = nrows - r0 < kUnpackRows ? nrows - r0 : kUnpackRows;
    for (int kk = ty; kk < 32; kk += 8) {
        const int k = kt * 32 + kk, l = lt * 32 + lane;
        if (k < nbf && l <= k) {
            const int64_t KL = (int64_t)k * (k + 1) / 2 + l, col = KL * (KL + 1) / 2 + IJ0;
#pragma unroll
            for (int r = 0; r < kUnpackRows; ++r) {
                const int64_t IJ = IJ0 + r;
                if (r < rows) s[r][kk][lane] = __ldg(ints + (KL <= IJ ? IJ * (IJ + 1) / 2 + KL : col + r));
            }
        }
    }
    __syncthreads();
    for (int r = 0; r < rows; ++r) {
        double *o = out + (int64_t)(r0 + r) * nbf * nbf;
        for (int kk = ty; kk < 32; kk += 8) {
            const int k = kt * 32 + kk, l = lt * 32 + lane;
            if (k < nbf && l < nbf) o[(int64_t)k * nbf + l] = lt < kt || lane <= kk ? s[r][kk][lane] : s[r][lane][kk];
            const int kT = lt * 32 + kk, lT = kt * 32 + lane;
            if (lt < kt && lT < nbf) o[(int64_t)kT * nbf + lT] = s[r][lane][kk];
        }
    }
}

// out[(mu * nbf + nu) * ncol + c] = Y[pair(mu, nu) * ncol + c].
__global__ void mo_unpack_pairs_kernel(const double *__restrict__ Y, int nbf, int64_t ncol, double *__restrict__ out)
{
    const int64_t total = (int64_t)nbf * nbf * ncol;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        const int64_t row = t / ncol, c = t - row * ncol;
        const int64_t mu = row / nbf, nu = row - mu * nbf;
        out[t] = __ldg(Y + pair_of(mu, nu) * ncol + c);
    }
}

// out[((a * nbf + nu) * nb + b) * nj + j] =
//     sum_mu C[mu * na + a] Y[(b * P + pair(mu, nu)) * nj + j],
// the contraction over one index of a symmetric pair (mu, nu) stored once, as
// FP64 tensor-core tiles: a block takes one nu, MT = 8 MF of the na columns of
// C and 64 of the nb * nj columns (b, j), and gathers the rows pair(mu, nu) of
// Y as its K dimension, so the pair index is never unpacked to nbf^2 rows.
// nu runs fastest over the grid: the P rows of a 64-column strip (5.8 MB at
// N = 150) stay in L2 for both orders of every pair.  N = 150, 30 columns of
// C, 3,600 of Y: 0.29 ms (16.5 TFLOP/s); the unpacked copy alone took 0.37 ms.
constexpr int kPairK = 16, kPairCols = 64, kPairStages = 3, kPairPitchB = kPairCols + 4;

template <int MF> struct PairLayout {
    static constexpr int MT = 8 * MF;
    static constexpr int pitchA = (MT + 15) / 16 * 16 + 4;   // 4 mod 16 doubles: fragment reads hit distinct banks
    static constexpr int stage = kPairK * (pitchA + kPairPitchB);
    static constexpr size_t bytes = sizeof(double) * kPairStages * stage;
};

template <int MF>
__global__ void __launch_bounds__(128) mo_contract_pairs_kernel(const double *__restrict__ Y, int nbf, int nb, int nj,
                                                                const double *__restrict__ C, int na,
                                                                double *__restrict__ out)
{
    using Lay = PairLayout<MF>;
    extern __shared__ double sm[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nu = blockIdx.x, a0 = blockIdx.z * Lay::MT;
    const int64_t P = (int64_t)nbf * (nbf + 1) / 2, ncol = (int64_t)nb * nj, c0 = (int64_t)blockIdx.y * kPairCols;
    // this thread's column of the B tile
    const int64_t cc = c0 + (tid & 63), cs = cc < ncol ? cc : 0;
    const double *Yc = Y + (cs / nj) * P * nj + cs % nj;
    auto load = [&](int k0, int slot) {
        double *As = sm + slot * Lay::stage, *Bs = As + kPairK * Lay::pitchA;
        for (int e = tid; e < kPairK * Lay::MT; e += 128) {
            const int k = e / Lay::MT, a = e - k * Lay::MT;
            const bool ok = k0 + k < nbf && a0 + a < na;
            cp_async8(As + k * Lay::pitchA + a, ok ? C + (int64_t)(k0 + k) * na + a0 + a : C, ok);
        }
#pragma unroll
        for (int k = tid >> 6; k < kPairK; k += 2) {
            const bool ok = k0 + k < nbf && cc < ncol;
            cp_async8(Bs + k * kPairPitchB + (tid & 63), ok ? Yc + pair_of(k0 + k, nu) * nj : Y, ok);
        }
    };
    double acc[MF][2][2];
#pragma unroll
    for (int m = 0; m < MF; ++m)
#pragma unroll
        for (int n = 0; n < 2; ++n) acc[m][n][0] = acc[m][n][1] = 0.0;
    const int nk = (nbf + kPairK - 1) / kPairK;
#pragma unroll
    for (int s = 0; s < kPairStages - 1; ++s) {
        if (s < nk) load(s * kPairK, s);
        cp_async_commit();
    }
    for (int t = 0; t < nk; ++t) {
        cp_async_wait<kPairStages - 2>();
        __syncthreads();   // stage t has landed; stage t - 1's readers are done
        if (t + kPairStages - 1 < nk) load((t + kPairStages - 1) * kPairK, (t + kPairStages - 1) % kPairStages);
        cp_async_commit();
        const double *As = sm + (t % kPairStages) * Lay::stage + (lane & 3) * Lay::pitchA + (lane >> 2);
        const double *Bs = sm + (t % kPairStages) * Lay::stage + kPairK * Lay::pitchA + (lane & 3) * kPairPitchB +
                           warp * 16 + (lane >> 2);
#pragma unroll
        for (int k = 0; k < kPairK; k += 4) {
            double b[2], a[MF];
#pragma unroll
            for (int n = 0; n < 2; ++n) b[n] = Bs[k * kPairPitchB + 8 * n];
#pragma unroll
            for (int m = 0; m < MF; ++m) a[m] = As[k * Lay::pitchA + 8 * m];
#pragma unroll
            for (int m = 0; m < MF; ++m)
#pragma unroll
                for (int n = 0; n < 2; ++n) dmma(acc[m][n], a[m], b[n]);
        }
    }
#pragma unroll
    for (int m = 0; m < MF; ++m)
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            const int a = a0 + 8 * m + (lane >> 2);
            const int64_t c = c0 + warp * 16 + 8 * n + 2 * (lane & 3);
            double *o = out + ((int64_t)a * nbf + nu) * ncol + c;
            if (a < na && c < ncol) o[0] = acc[m][n][0];
            if (a < na && c + 1 < ncol) o[1] = acc[m][n][1];
        }
}

template <int MF>
cudaError_t launch_contract_pairs(const double *Y, int nbf, int nb, int nj, const double *C, int na, double *out, int nz,
                                  cudaStream_t st)
{
    using Lay = PairLayout<MF>;
    const cudaError_t e = cudaFuncSetAttribute(mo_contract_pairs_kernel<MF>,
                                               cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Lay::bytes);
    if (e != cudaSuccess) return e;
    const int64_t strips = ((int64_t)nb * nj + kPairCols - 1) / kPairCols;
    // (the grid's y dimension holds 65535 strips a launch: 4.2 M columns, more than Y's rows fit in memory for)
    if (strips > 65535) return cudaErrorInvalidValue;
    mo_contract_pairs_kernel<MF><<<dim3(nbf, (unsigned)strips, nz), 128, Lay::bytes, st>>>(Y, nbf, nb, nj, C, na, out);
    return cudaGetLastError();
}

// out[(b * nrows + r) * nbf + l] = sum_k C[k * nb + b] (IJ_r|kl), IJ_r = row0 + r:
// the first quarter transformation straight from the packed order, as FP64
// tensor-core tiles.  A block takes four consecutive bra rows IJ, whose neighbouring
// numbers fill the 32-byte sectors where a later row holds them (kl > IJ), and
// streams the panels of eight k through shared memory, three in flight; the
// products of the whole pass (for example 160 l, 32 b for each row) stay in
// registers, RT x 2 tiles a warp, so no unpacked row is ever written.  A panel's
// 8 x 8 part with l >= k is copied along k, the others along l, whichever is
// contiguous in the packed row.  Each number is read twice (for k and for l),
// from L2 the second time.
// N = 150, 30 columns, all 11,325 rows: 0.91 ms (16.8 TFLOP/s); unpacking (0.95 ms) and a library
// product (0.71 ms) before.  (One row a block, kept whole in shared memory, read
// one number per sector: 1.9 ms.)
constexpr int kRowsGroup = 4, kRowsStages = 3, kRowsThreads = 512;

// How the 16 warps share a pass: each row has `sgroups` warps along l, RT strips of
// 8 each, and 4 / sgroups along b, two tiles each.
struct RowsLayout {
    int rt, sgroups, cgroups, spasses, cpasses, pitch, row, pitchC, stage;
    size_t bytes;
    RowsLayout(int nbf, int nb) : rt(0)
    {
        const int strips = (nbf + 7) / 8, pairs = (nb + 15) / 16;
        int64_t best = 0;
        for (int sg = 1; sg <= 4; sg *= 2) {
            // (four times nine strips are what shared memory holds, ten what the registers do)
            const int most = (sg == 4 ? 9 : 10) * sg;
            const int cg = 4 / sg, sp = (strips + most - 1) / most, cp = (pairs + cg - 1) / cg;
            const int t = (strips + sp * sg - 1) / (sp * sg);
            const int64_t cost = (int64_t)sp * cp * (t + 1);   // a warp's tiles, and its share of the panels' traffic
            if (rt == 0 || cost < best) {
                best = cost;
                rt = t, sgroups = sg, cgroups = cg, spasses = sp, cpasses = cp;
            }
        }
        pitch = 8 * rt * sgroups + 4;       // 4 or 12 mod 16 doubles: fragment reads hit distinct banks
        row = 8 * pitch + 5;                // the copies' four rows likewise
        pitchC = 16 * cgroups + 4;
        stage = kRowsGroup * row + 8 * pitchC;
        bytes = sizeof(double) * kRowsStages * stage;
    }
};

template <int RT>
__global__ void __launch_bounds__(kRowsThreads) mo_contract_rows_kernel(const double *__restrict__ ints, int nbf,
                                                                        int64_t row0, int nrows,
                                                                        const double *__restrict__ C, int nb,
                                                                        RowsLayout lay, double *__restrict__ out)
{
    extern __shared__ double sm[];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, c = lane & 3, r8 = lane >> 2;
    const int panels = (nbf + 7) / 8, nstrip = RT * lay.sgroups;
    const int S0 = blockIdx.y % lay.spasses * nstrip, b0 = blockIdx.y / lay.spasses * 16 * lay.cgroups;
    const int groups = (nrows + kRowsGroup - 1) / kRowsGroup;
    const int cshift = 4 + (lay.cgroups >> 1);   // 16 cgroups columns, cgroups 1, 2 or 4
    // Copies: a lane's row is c; a warp's instruction takes line `warp % 8` of an 8 x 8 part, eight numbers by four
    // rows.  (32-bit pair indices, one 64-bit product for a later row's number: the addresses are what these cost.)
    auto fetch = [&](int g, int K, double *A) {
        const int r = g * kRowsGroup + c;
        const bool row_ok = r < nrows;
        const unsigned IJ = (unsigned)row0 + (row_ok ? r : 0);
        const double *const base = ints + (uint64_t)IJ * (IJ + 1) / 2, *const col = ints + IJ;
        double *const Ar = A + c * lay.row;
        const int s = warp & 7;
        auto one = [&](int k, int l, int hi, int lo) {
            const unsigned q = (unsigned)(hi * (hi + 1)) / 2 + lo;
            const double *const src = q <= IJ ? base + q : (const double *)((const char *)col + 4 * ((uint64_t)q * (q + 1)));
            const bool ok = row_ok && hi < nbf;
            cp_async8(Ar + (k & 7) * lay.pitch + l - 8 * S0, ok ? src : ints, ok);
        };
        int L = S0 + (warp >> 3);
        const int end = S0 + nstrip;
#pragma unroll 2
        for (; L < K && L < end; L += 2) one(8 * K + s, 8 * L + r8, 8 * K + s, 8 * L + r8);
#pragma unroll 2
        for (; L < end; L += 2) {
            const int l = 8 * L + s, k = 8 * K + r8;
            one(k, l, max(k, l), min(k, l));
        }
        double *const Cs = A + kRowsGroup * lay.row;
        for (int e = tid; e < 8 << cshift; e += kRowsThreads) {
            const int k = e >> cshift, b = e & ((1 << cshift) - 1);
            const bool ok = 8 * K + k < nbf && b0 + b < nb;
            cp_async8(Cs + k * lay.pitchC + b, ok ? C + (int64_t)(8 * K + k) * nb + b0 + b : C, ok);
        }
    };
    // this warp's row and tiles
    const int rw = warp & 3, sg = (warp >> 2) % lay.sgroups, cg = (warp >> 2) / lay.sgroups;
    const double *const Af = sm + rw * lay.row + c * lay.pitch + 8 * RT * sg + r8;
    const double *const Cf = sm + kRowsGroup * lay.row + c * lay.pitchC + 16 * cg + r8;
    double acc[RT][2][2];
#pragma unroll
    for (int t = 0; t < RT; ++t)
#pragma unroll
        for (int n = 0; n < 2; ++n) acc[t][n][0] = acc[t][n][1] = 0.0;
    // one stream of panels over all the block's row groups
    int gl = blockIdx.x, Kl = 0, slot = 0;
    const bool early = (warp >> 2 & 1) == 0;
    auto next = [&](int sl) {
        if (gl < groups) {
            fetch(gl, Kl, sm + sl * lay.stage);
            if (++Kl == panels) Kl = 0, gl += gridDim.x;
        }
        cp_async_commit();
    };
#pragma unroll
    for (int s = 0; s < kRowsStages - 1; ++s) next(s);
    for (int g = blockIdx.x; g < groups; g += gridDim.x) {
        for (int K = 0; K < panels; ++K) {
            cp_async_wait<kRowsStages - 2>();
            __syncthreads();   // this panel has landed; the last one's readers are done
            // half of each scheduler's warps copy while the others multiply
            const int into = slot == 0 ? kRowsStages - 1 : slot - 1;
            if (early) next(into);
            const double *const As = Af + slot * lay.stage, *const Cs = Cf + slot * lay.stage;
#pragma unroll
            for (int k = 0; k < 8; k += 4) {
                const double a0 = Cs[k * lay.pitchC], a1 = Cs[k * lay.pitchC + 8];
#pragma unroll
                for (int t = 0; t < RT; ++t) {
                    const double v = As[k * lay.pitch + 8 * t];
                    dmma(acc[t][0], a0, v);
                    dmma(acc[t][1], a1, v);
                }
            }
            if (!early) next(into);
            slot = slot + 1 == kRowsStages ? 0 : slot + 1;
        }
        const int r = g * kRowsGroup + rw;
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            const int b = b0 + 16 * cg + 8 * n + r8;
            double *const o = out + ((int64_t)b * nrows + r) * nbf;
#pragma unroll
            for (int t = 0; t < RT; ++t) {
                const int l = 8 * (S0 + RT * sg + t) + 2 * c;
                if (r < nrows && b < nb && l < nbf) o[l] = acc[t][n][0];
                if (r < nrows && b < nb && l + 1 < nbf) o[l + 1] = acc[t][n][1];
                acc[t][n][0] = acc[t][n][1] = 0.0;
            }
        }
    }
}

template <int RT>
cudaError_t launch_contract_rows(const double *ints, int nbf, int64_t row0, int nrows, const double *C, int nb,
                                 const RowsLayout &lay, double *out, cudaStream_t st)
{
    const auto kernel = mo_contract_rows_kernel<RT>;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)lay.bytes);
    int dev = 0, nsm = 0, per = 0;
    if (e == cudaSuccess) e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, kRowsThreads, lay.bytes);
    if (e != cudaSuccess) return e;
    const int passes = lay.spasses * lay.cpasses, groups = (nrows + kRowsGroup - 1) / kRowsGroup;
    if (passes > 65535) return cudaErrorInvalidValue;
    const int resident = nsm * (per > 0 ? per : 1) / passes;
    const int grid = resident < 1 ? 1 : resident < groups ? resident : groups;
    kernel<<<dim3(grid, passes), kRowsThreads, lay.bytes, st>>>(ints, nbf, row0, nrows, C, nb, lay, out);
    return cudaGetLastError();
}

// moints[ijkl2intindex(a, i, b, j)] = Z[((a * nmo + i) * nocc + b) * nmo + j]
// for a, b < nocc, i, j < nmo.  Slots that several (a, i, b, j) share by
// symmetry receive the same integral.
__global__ void mo_pack_kernel(const double *__restrict__ Z, int nocc, int nmo, double *__restrict__ moints)
{
    const int64_t total = (int64_t)nocc * nmo * nocc * nmo;
    for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
        int64_t q = t;
        const int64_t j = q % nmo;
        q /= nmo;
        const int64_t b = q % nocc;
        q /= nocc;
        const int64_t i = q % nmo, a = q / nmo;
        moints[packed_of(pair_of(a, i), pair_of(b, j))] = Z[t];
    }
}

// One block per occupied pair (a, b): V[((a * nv + r) * nocc + b) * nv + s]
// = (ar|bs) over the virtual orbitals r, s.
__global__ void __launch_bounds__(256) mp2_pairs_kernel(const double *__restrict__ V, int nocc, int nv,
                                                        const double *__restrict__ e_occ,
                                                        const double *__restrict__ e_virt, double *__restrict__ Epair)
{
    const int a = blockIdx.x / nocc, b = blockIdx.x - a * nocc;
    const double eab = e_occ[a] + e_occ[b];
    double sum = 0.0;
    for (int t = threadIdx.x; t < nv * nv; t += blockDim.x) {
        const int r = t / nv, s = t - r * nv;
        const double v = V[(((int64_t)a * nv + r) * nocc + b) * nv + s];
        const double w = V[(((int64_t)a * nv + s) * nocc + b) * nv + r];
        sum += v * (2.0 * v - w) / (eab - e_virt[r] - e_virt[s]);
    }
    __shared__ double red[32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = sum;
    __syncthreads();
    if (threadIdx.x < 32) {
        sum = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, o);
        if (threadIdx.x == 0) Epair[blockIdx.x] = sum;
    }
}

int grid_for(int64_t total)
{
    const int64_t g = (total + 255) / 256;
    return (int)(g < 148 * 32 ? (g > 0 ? g : 1) : 148 * 32);
}

}  // namespace

extern "C" {

int pqb_mo_unpack_rows(const double *ints, int64_t len, int nbf, int64_t row0, int nrows, double *out, void *stream)
{
    if (!ints || !out || nbf <= 0 || nrows <= 0 || row0 < 0) return PQB_E_ARG;
    const int64_t P = (int64_t)nbf * (nbf + 1) / 2;
    if (len != P * (P + 1) / 2 || row0 + nrows > P) return PQB_E_SHAPE;
    const int nt = (nbf + 31) / 32, nt2 = nt * (nt + 1) / 2;
    // (at most 2^31 - 1 blocks a launch)
    const int64_t groups = ((int64_t)nrows + kUnpackRows - 1) / kUnpackRows, most = 0x7fffffff / nt2;
    for (int64_t g = 0; g < groups; g += most) {
        const int64_t r = g * kUnpackRows, ng = groups - g < most ? groups - g : most;
        const int64_t left = nrows - r < ng * kUnpackRows ? nrows - r : ng * kUnpackRows;
        mo_unpack_rows_kernel<<<(unsigned)(ng * nt2), 256, 0, (cudaStream_t)stream>>>(ints, nbf, row0 + r, (int)left, nt2,
                                                                                      out + r * nbf * nbf);
    }
    return cudaGetLastError() == cudaSuccess ? PQB_OK : PQB_E_CUDA;
}

int pqb_mo_unpack_pairs(const double *Y, int nbf, int64_t ncol, double *out, void *stream)
{
    if (!Y || !out || nbf <= 0 || ncol <= 0) return PQB_E_ARG;
    const int64_t total = (int64_t)nbf * nbf * ncol;
    mo_unpack_pairs_kernel<<<grid_for(total), 256, 0, (cudaStream_t)stream>>>(Y, nbf, ncol, out);
    return cudaGetLastError() == cudaSuccess ? PQB_OK : PQB_E_CUDA;
}

int pqb_mo_contract_pairs(const double *Y, int nbf, int nb, int nj, const double *C, int na, double *out, void *stream)
{
    if (!Y || !C || !out || nbf <= 0 || nb <= 0 || nj <= 0 || na <= 0) return PQB_E_ARG;
    // rows of C a block: all of them up to 64, else equal parts
    const int nz = (na + 63) / 64, mf = ((na + nz - 1) / nz + 7) / 8;
    cudaStream_t st = (cudaStream_t)stream;
    cudaError_t e = cudaErrorInvalidValue;
    switch (mf) {
    case 1: e = launch_contract_pairs<1>(Y, nbf, nb, nj, C, na, out, nz, st); break;
    case 2: e = launch_contract_pairs<2>(Y, nbf, nb, nj, C, na, out, nz, st); break;
    case 3: e = launch_contract_pairs<3>(Y, nbf, nb, nj, C, na, out, nz, st); break;
    case 4: e = launch_contract_pairs<4>(Y, nbf, nb, nj, C, na, out, nz, st); break;
    case 5: e = launch_contract_pairs<5>(Y, nbf, nb, nj, C, na, out, nz, st); break;
    case 6: e = launch_contract_pairs<6>(Y, nbf, nb, nj, C, na, out, nz, st); break;
    case 7: e = launch_contract_pairs<7>(Y, nbf, nb, nj, C, na, out, nz, st); break;
    case 8: e = launch_contract_pairs<8>(Y, nbf, nb, nj, C, na, out, nz, st); break;
    }
    return e == cudaSuccess ? PQB_OK : PQB_E_CUDA;
}

int pqb_mo_contract_rows(const double *ints, int64_t len, int nbf, int64_t row0, int nrows, const double *C, int nb,
                         double *out, void *stream)
{
    if (!ints || !C || !out || nbf <= 0 || nb <= 0 || nrows <= 0 || row0 < 0) return PQB_E_ARG;
    const int64_t P = (int64_t)nbf * (nbf + 1) / 2;
    if (len != P * (P + 1) / 2 || row0 + nrows > P) return PQB_E_SHAPE;
    const RowsLayout lay(nbf, nb);
    cudaStream_t st = (cudaStream_t)stream;
    cudaError_t e = cudaErrorInvalidValue;
    switch (lay.rt) {
    case 1: e = launch_contract_rows<1>(ints, nbf, row0, nrows, C, nb, lay, out, st); break;
    case 2: e = launch_contract_rows<2>(ints, nbf, row0, nrows, C, nb, lay, out, st); break;
    case 3: e = launch_contract_rows<3>(ints, nbf, row0, nrows, C, nb, lay, out, st); break;
    case 4: e = launch_contract_rows<4>(ints, nbf, row0, nrows, C, nb, lay, out, st); break;
    case 5: e = launch_contract_rows<5>(ints, nbf, row0, nrows, C, nb, lay, out, st); break;
    case 6: e = launch_contract_rows<6>(ints, nbf, row0, nrows, C, nb, lay, out, st); break;
    case 7: e = launch_contract_rows<7>(ints, nbf, row0, nrows, C, nb, lay, out, st); break;
    case 8: e = launch_contract_rows<8>(ints, nbf, row0, nrows, C, nb, lay, out, st); break;
    case 9: e = launch_contract_rows<9>(ints, nbf, row0, nrows, C, nb, lay, out, st); break;
    case 10: e = launch_contract_rows<10>(ints, nbf, row0, nrows, C, nb, lay, out, st); break;
    }
    return e == cudaSuccess ? PQB_OK : PQB_E_CUDA;
}

int pqb_mo_pack(const double *Z, int nocc, int nmo, double *moints, int64_t len, void *stream)
{
    if (!Z || !moints || nocc <= 0 || nmo <= 0 || nocc > nmo) return PQB_E_ARG;
    const int64_t P = (int64_t)nmo * (nmo + 1) / 2;
    if (len != P * (P + 1) / 2) return PQB_E_SHAPE;
    const int64_t total = (int64_t)nocc * nmo * nocc * nmo;
    mo_pack_kernel<<<grid_for(total), 256, 0, (cudaStream_t)stream>>>(Z, nocc, nmo, moints);
    return cudaGetLastError() == cudaSuccess ? PQB_OK : PQB_E_CUDA;
}

int pqb_mp2_pairs(const double *V, int nocc, int nvirt, const double *e_occ, const double *e_virt, double *Epair,
                  void *stream)
{
    if (!V || !e_occ || !e_virt || !Epair || nocc <= 0 || nvirt < 0) return PQB_E_ARG;
    if (nvirt == 0) return cudaMemsetAsync(Epair, 0, sizeof(double) * nocc * nocc, (cudaStream_t)stream) ==
                                   cudaSuccess ? PQB_OK : PQB_E_CUDA;
    mp2_pairs_kernel<<<nocc * nocc, 256, 0, (cudaStream_t)stream>>>(V, nocc, nvirt, e_occ, e_virt, Epair);
    return cudaGetLastError() == cudaSuccess ? PQB_OK : PQB_E_CUDA;
}

}  // extern "C"
