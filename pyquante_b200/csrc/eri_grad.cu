// Nuclear gradient of the two-electron energy, contracted on the fly:
//
//   dE2/dX = sum over unique (ij|kl) of  d(ij|kl)/dX * Gamma_ijkl,
//   Gamma_ijkl = 8 s (2 D_ij D_kl - (D_ik D_jl + D_il D_jk)/2),
//
// s the 8-fold degeneracy weight (1/2 per i==j, k==l, ij==kl), which is
// E2 = sum_ijkl (ij|kl)(2 D_ij D_kl - D_ik D_jl) of the RHF energy
// E = tr(D h) + tr(D F) (PyQuante/hartree_fock.py:33-38) differentiated; the
// reference forms it as trace2(D, der2JmK(...)) over stored derivative
// integrals (PyQuante/force.py:106-116,232-252,318-357).
//
// Derivative integrals come from the Rys 2-D integrals with one more unit of
// momentum on centres A and C,
//   d/dA_x phi_a = 2 alpha_a phi_{a+1x} - a_x phi_{a-1x}
// (the raising/lowering relation of PyQuante/AnalyticDerivatives.py, applied
// to each primitive), the raised B from the horizontal relation
// (a,b+1) = (a+1,b) + AB (a,b), and the fourth centre by translational
// invariance, dD = -(dA + dB + dC).
//
// The components are those of the shells' common contraction: D is the
// pre-scaled density D'_kl = r_k r_l D_kl of the Fock-build kernels, so Gamma
// carries the four component scales.  The gradient is summed per shell
// in kGradCopies sets of 3 nshell accumulators, one set per block in turn, and
// gathered to the atoms at the end.  A single set has every item of a build add
// to the same few hundred numbers, one after the other in L2: C5H12 / 6-31G* 3.15
// -> 1.46 ms, C10H22 / STO-3G 2.77 -> 0.96, C8H18 / 6-31G** 16.0 -> 10.1 with 64.
//
// Two splits (eri_grad_launch picks by the number of components):
//  * up to 27 components: one thread per work item, everything in registers;
//  * more: one warp per work item.  Lanes first share the (primitive quartet,
//    root, axis) 2-D tables, which go to shared memory, then the (component,
//    root) products.
// (H2O)4 / 6-31G* takes 185 us on the GPU (0.31 ms with one set of sums; 50 ms
// with one thread per item for every class, its tables and Gamma in local memory,
// and the classes one after the other): the items' serial chains and the few high
// classes leave most of the chip idle.  Four or eight lanes an item for up to 27
// components: slower at every size (Gamma is then fetched by each).
#include "eri_engine.cuh"
#include "eri_launch.h"

namespace pqb {

// Gamma of component (ia ib|ic id) without the weight, D' read at the
// quartet's functions.
__device__ __forceinline__ double gamma_of(const double *Db, int64_t nm, int i, int j, int k, int l)
{
    const double dij = __ldg(Db + i * nm + j), dkl = __ldg(Db + k * nm + l);
    const double dik = __ldg(Db + i * nm + k), djl = __ldg(Db + j * nm + l);
    const double dil = __ldg(Db + i * nm + l), djk = __ldg(Db + j * nm + k);
    return 16.0 * dij * dkl - 4.0 * (dik * djl + dil * djk);
}

// ---------------------------------------------------------- thread mode --
template <int LA, int LB, int LC, int LD>
__global__ void __launch_bounds__(128) eri_grad_thread_kernel(const int4 *__restrict__ list, int nq,
                                                              const PairInfo *__restrict__ pairs,
                                                              const PrimPair *__restrict__ prims,
                                                              const double *__restrict__ D, double *gshell, int glen)
{
    gshell += (int64_t)(blockIdx.x % kGradCopies) * glen;   // this block's copy of the sums
    constexpr int NA = ncart(LA), NB = ncart(LB), NC = ncart(LC), ND = ncart(LD);
    constexpr int NR = (LA + LB + LC + LD + 1) / 2 + 1;
    constexpr int sD = 1, sC = (LD + 1) * sD, sB = (LC + 2) * sC, sA = (LB + 1) * sB, G2 = (LA + 2) * sA;
    const int lane = threadIdx.x & 31;
    // whole warps step through the list; a lane past the end repeats the last
    // item with no primitive quartets
    for (int base = blockIdx.x * blockDim.x + threadIdx.x - lane; base < nq; base += gridDim.x * blockDim.x) {
        const int qi = base + lane;
        const bool live = qi < nq;
        const int4 e = list[live ? qi : nq - 1];
        const PairInfo &pb = pairs[e.x];
        const PairInfo &pk = pairs[e.y];
        const QCtx q = make_qctx(pb, pk, e.x, e.y);
        const bool bd = q.sa == q.sb, kd = q.sc == q.sd, qd = q.bra == q.ket, af = q.fa > q.fb;
        const double *Db = D + q.bo;
        double gam[NA * NB * NC * ND];
#pragma unroll
        for (int a = 0; a < NA; ++a)
#pragma unroll
            for (int b = 0; b < NB; ++b)
#pragma unroll
                for (int c = 0; c < NC; ++c)
#pragma unroll
                    for (int d = 0; d < ND; ++d)
                        gam[((a * NB + b) * NC + c) * ND + d] =
                            comp_weight(a, b, c, d, bd, kd, qd, af) *
                            gamma_of(Db, q.nm, q.fa + a, q.fb + b, q.fc + c, q.fd + d);
        double g9[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) g9[k] = 0.0;
        const double AB[3] = {pb.AB[0], pb.AB[1], pb.AB[2]}, CD[3] = {pk.AB[0], pk.AB[1], pk.AB[2]};
        const double A[3] = {pb.A[0], pb.A[1], pb.A[2]}, C[3] = {pk.A[0], pk.A[1], pk.A[2]};
        // bra primitives fastest: the lanes of a warp mostly share the bra pair
        const int npb = pb.nprim;
        int ik = e.z / npb, ib = e.z - (e.z / npb) * npb;
        const int count = live ? e.w : 0;
#pragma unroll 1
        for (int t = 0; t < count; ++t) {
            const PrimPair *pp = prims + pb.prim_off + ib, *pq = prims + pk.prim_off + ik;
            const PrimJK P = load_prim_jk(pp), Q = load_prim_jk(pq);
            const double a2 = 2.0 * __ldg(&pp->alpha_a), b2 = 2.0 * P.zeta - a2, c2 = 2.0 * __ldg(&pq->alpha_a);
            if (++ib == npb) {
                ib = 0;
                ++ik;
            }
            const double PQ[3] = {P.P[0] - Q.P[0], P.P[1] - Q.P[1], P.P[2] - Q.P[2]};
            const double rs = rsqrt_nr(P.zeta + Q.zeta), izpe = rs * rs;
            const double T = P.zeta * Q.zeta * izpe * (PQ[0] * PQ[0] + PQ[1] * PQ[1] + PQ[2] * PQ[2]);
            const double pre = P.K * Q.K * rs;
            double uu[NR], ww[NR];
            rys_roots_fast<NR>(T, uu, ww);
#pragma unroll
            for (int r = 0; r < NR; ++r) {
                const RysCoef k = rys_coef(uu[r], P.zeta, Q.zeta, P.izeta, Q.izeta, izpe);
                double g[3][G2];
#pragma unroll
                for (int x = 0; x < 3; ++x)
                    rys2d_c<LA + 1, LB, LC + 1, LD, double>(k, P.P[x] - A[x], Q.P[x] - C[x], PQ[x], AB[x], CD[x],
                                                            x == 0 ? ww[r] * pre : 1.0, g[x]);
#pragma unroll
                for (int ab = 0; ab < NA * NB; ++ab)
#pragma unroll
                    for (int cd = 0; cd < NC * ND; ++cd) {
                        const int ia = ab / NB, ib3 = ab % NB, ic = cd / ND, id = cd % ND;
                        double I[3], dA[3], dB[3], dC[3];
#pragma unroll
                        for (int x = 0; x < 3; ++x) {
                            const int a = cart_l(LA, ia, x), b = cart_l(LB, ib3, x), c = cart_l(LC, ic, x),
                                      d = cart_l(LD, id, x);
                            const int o = a * sA + b * sB + c * sC + d * sD;
                            const double up = g[x][o + sA];
                            I[x] = g[x][o];
                            dA[x] = a2 * up - (a > 0 ? a * g[x][o - (a > 0 ? sA : 0)] : 0.0);
                            dB[x] = b2 * fma(AB[x], I[x], up) - (b > 0 ? b * g[x][o - (b > 0 ? sB : 0)] : 0.0);
                            dC[x] = c2 * g[x][o + sC] - (c > 0 ? c * g[x][o - (c > 0 ? sC : 0)] : 0.0);
                        }
                        const double gm = gam[ab * NC * ND + cd];
                        const double w0 = gm * I[1] * I[2], gx = gm * I[0], w1 = gx * I[2], w2 = gx * I[1];
                        g9[0] = fma(w0, dA[0], g9[0]);
                        g9[1] = fma(w1, dA[1], g9[1]);
                        g9[2] = fma(w2, dA[2], g9[2]);
                        g9[3] = fma(w0, dB[0], g9[3]);
                        g9[4] = fma(w1, dB[1], g9[4]);
                        g9[5] = fma(w2, dB[2], g9[5]);
                        g9[6] = fma(w0, dC[0], g9[6]);
                        g9[7] = fma(w1, dC[1], g9[7]);
                        g9[8] = fma(w2, dC[2], g9[8]);
                    }
            }
        }
        // last shell: one atomic per lane (neighbouring items differ in it); third:
        // one per run of lanes that share it; bra shells: one per warp while the
        // warp holds one bra pair (the item order is bra-major), else per run
        const WarpRuns rbc(q.bra, q.sc, lane);
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            if (count > 0) atomicAdd(gshell + 3 * q.sd + x, -(g9[x] + g9[3 + x] + g9[6 + x]));
            const double s = rbc.sum(g9[6 + x]);
            if (rbc.last) atomicAdd(gshell + 3 * q.sc + x, s);
        }
        const int bra0 = __shfl_sync(0xffffffffu, q.bra, 0);
        const bool one_bra = __all_sync(0xffffffffu, bra0 == q.bra);
        if (one_bra) {
            int idx;
            const double s = warp_sum_transposed<6>(g9, lane, idx);
            if (idx < 6 && (lane & 3) == 0) atomicAdd(gshell + 3 * (idx < 3 ? q.sa : q.sb) + idx % 3, s);
        } else {
            const WarpRuns rb(q.bra, 0, lane);
#pragma unroll
            for (int x = 0; x < 3; ++x) {
                const double sa = rb.sum(g9[x]), sb = rb.sum(g9[3 + x]);
                if (rb.last) {
                    atomicAdd(gshell + 3 * q.sa + x, sa);
                    atomicAdd(gshell + 3 * q.sb + x, sb);
                }
            }
        }
    }
}

// ------------------------------------------------------------ warp mode --
template <int LA, int LB, int LC, int LD> struct GradWarpLayout {
    static constexpr int NCOMP = ncart(LA) * ncart(LB) * ncart(LC) * ncart(LD);
    static constexpr int NR = (LA + LB + LC + LD + 1) / 2 + 1;
    static constexpr int sC = LD + 1, sB = (LC + 2) * sC, sA = (LB + 1) * sB, G2 = (LA + 2) * sA;
    // an odd pitch spreads the (root, axis) tables over the banks
    static constexpr int pitch = G2 | 1;
    static constexpr size_t pq_bytes = sizeof(double) * 3 * NR * pitch;
    // primitive quartets of one pass: their (root, axis) tables occupy the
    // lanes, within 16 KB of tables a warp
    static constexpr int fit = 32 / (3 * NR);
    static constexpr int PB = fit > 1 && pq_bytes * fit <= 16384 ? fit : (fit > 2 && pq_bytes * 2 <= 16384 ? 2 : 1);
    static constexpr size_t warp_bytes = PB * pq_bytes + sizeof(double) * NCOMP;
    static constexpr int warps = 4 * warp_bytes + sizeof(uint2) * NCOMP <= 56 * 1024 ? 4 : 2;
    static constexpr size_t bytes = warps * warp_bytes + sizeof(uint2) * NCOMP;
};

// One warp per item.  Bound by shared-memory wavefronts (18 loads per
// component and root for about 36 FP64 operations; neighbouring lanes'
// components share most of them).
template <int LA, int LB, int LC, int LD>
__global__ void __launch_bounds__(GradWarpLayout<LA, LB, LC, LD>::warps * 32)
eri_grad_warp_kernel(const int4 *__restrict__ list, int nq, const PairInfo *__restrict__ pairs,
                     const PrimPair *__restrict__ prims, const double *__restrict__ D, double *gshell, int glen)
{
    gshell += (int64_t)(blockIdx.x % kGradCopies) * glen;   // this block's copy of the sums
    using Lay = GradWarpLayout<LA, LB, LC, LD>;
    constexpr int NA = ncart(LA), NB = ncart(LB), NC = ncart(LC), ND = ncart(LD), NCD = NC * ND;
    constexpr int NR = Lay::NR, NCOMP = Lay::NCOMP, PB = Lay::PB, PITCH = Lay::pitch, W = Lay::warps;
    constexpr int sA = Lay::sA, sB = Lay::sB, sC = Lay::sC;
    extern __shared__ __align__(16) unsigned char gsm[];
    __shared__ double expo[W][PB][3];   // 2 alpha_a, 2 alpha_b, 2 alpha_c of the pass
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double *tab = reinterpret_cast<double *>(gsm) + (size_t)warp * (Lay::warp_bytes / sizeof(double));
    double *gam = tab + PB * 3 * NR * PITCH;
    // per component: offsets of its x, y, z factors and the lowered powers
    uint2 *meta = reinterpret_cast<uint2 *>(gsm + W * Lay::warp_bytes);
    for (int t = threadIdx.x; t < NCOMP; t += W * 32) {
        const int ab = t / NCD, cd = t - ab * NCD;
        unsigned off[3], pw = 0;
        for (int x = 0; x < 3; ++x) {
            const int a = cart_l(LA, ab / NB, x), b = cart_l(LB, ab % NB, x), c = cart_l(LC, cd / ND, x),
                      d = cart_l(LD, cd % ND, x);
            off[x] = a * sA + b * sB + c * sC + d;
            pw |= (unsigned)(a | (b << 2) | (c << 4)) << (6 * x);
        }
        meta[t] = make_uint2(off[0] | (off[1] << 10) | (off[2] << 20), pw);
    }
    __syncthreads();
    for (int qi = blockIdx.x * W + warp; qi < nq; qi += gridDim.x * W) {
        const int4 e = list[qi];
        const PairInfo &pb = pairs[e.x];
        const PairInfo &pk = pairs[e.y];
        const QCtx q = make_qctx(pb, pk, e.x, e.y);
        const bool bd = q.sa == q.sb, kd = q.sc == q.sd, qd = q.bra == q.ket, af = q.fa > q.fb;
        const double *Db = D + q.bo;
        for (int t = lane; t < NCOMP; t += 32) {
            const int ab = t / NCD, cd = t - ab * NCD, ia = ab / NB, ib = ab % NB, ic = cd / ND, id = cd % ND;
            gam[t] = comp_weight(ia, ib, ic, id, bd, kd, qd, af) *
                     gamma_of(Db, q.nm, q.fa + ia, q.fb + ib, q.fc + ic, q.fd + id);
        }
        double g9[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) g9[k] = 0.0;
        const double AB[3] = {pb.AB[0], pb.AB[1], pb.AB[2]};
        const int npb = pb.nprim;
        for (int p0 = 0; p0 < e.w; p0 += PB) {
            const int nb = e.w - p0 < PB ? e.w - p0 : PB;
            __syncwarp();   // the tables of the pass before are read; gam is written
            if (lane < nb * 3 * NR) {
                const int b = lane / (3 * NR), rx = lane - b * (3 * NR), r = rx / 3, x = rx - r * 3;
                const int g = e.z + p0 + b, ik = g / npb, ib = g - ik * npb;
                const PrimPair *pp = prims + pb.prim_off + ib, *pq = prims + pk.prim_off + ik;
                const PrimJK P = load_prim_jk(pp), Q = load_prim_jk(pq);
                const double PQ[3] = {P.P[0] - Q.P[0], P.P[1] - Q.P[1], P.P[2] - Q.P[2]};
                const double rs = rsqrt_nr(P.zeta + Q.zeta), izpe = rs * rs;
                const double T = P.zeta * Q.zeta * izpe * (PQ[0] * PQ[0] + PQ[1] * PQ[1] + PQ[2] * PQ[2]);
                double u, w;
                rys_root(NR, r, T, u, w);
                const RysCoef k = rys_coef(u, P.zeta, Q.zeta, P.izeta, Q.izeta, izpe);
                const double Px = x == 0 ? P.P[0] : (x == 1 ? P.P[1] : P.P[2]);
                const double Qx = x == 0 ? Q.P[0] : (x == 1 ? Q.P[1] : Q.P[2]);
                rys2d_c<LA + 1, LB, LC + 1, LD, double>(k, Px - pb.A[x], Qx - pk.A[x], Px - Qx, pb.AB[x], pk.AB[x],
                                                        x == 0 ? w * P.K * Q.K * rs : 1.0, tab + lane * PITCH);
                if (rx == 0) {
                    const double a2 = 2.0 * __ldg(&pp->alpha_a);
                    expo[warp][b][0] = a2;
                    expo[warp][b][1] = 2.0 * P.zeta - a2;
                    expo[warp][b][2] = 2.0 * __ldg(&pq->alpha_a);
                }
            }
            __syncwarp();
            for (int t = lane; t < nb * NR * NCOMP; t += 32) {
                const int br = t / NCOMP, comp = t - br * NCOMP, b = br / NR;
                const double gm = gam[comp];
                if (gm == 0.0) continue;
                const uint2 m = meta[comp];
                const double a2 = expo[warp][b][0], b2 = expo[warp][b][1], c2 = expo[warp][b][2];
                double I[3], dA[3], dB[3], dC[3];
#pragma unroll
                for (int x = 0; x < 3; ++x) {
                    const double *g = tab + (br * 3 + x) * PITCH + ((m.x >> (10 * x)) & 1023u);
                    const int pw = m.y >> (6 * x), a = pw & 3, b1 = (pw >> 2) & 3, c = (pw >> 4) & 3;
                    const double up = g[sA];
                    I[x] = g[0];
                    // (a lowered power of zero multiplies the entry itself by zero)
                    dA[x] = fma(a2, up, -(double)a * g[a ? -sA : 0]);
                    dB[x] = fma(b2, fma(AB[x], I[x], up), LB > 0 ? -(double)b1 * g[b1 ? -sB : 0] : 0.0);
                    dC[x] = fma(c2, g[sC], LC > 0 ? -(double)c * g[c ? -sC : 0] : 0.0);
                }
                const double w0 = gm * I[1] * I[2], gx = gm * I[0], w1 = gx * I[2], w2 = gx * I[1];
                g9[0] = fma(w0, dA[0], g9[0]);
                g9[1] = fma(w1, dA[1], g9[1]);
                g9[2] = fma(w2, dA[2], g9[2]);
                g9[3] = fma(w0, dB[0], g9[3]);
                g9[4] = fma(w1, dB[1], g9[4]);
                g9[5] = fma(w2, dB[2], g9[5]);
                g9[6] = fma(w0, dC[0], g9[6]);
                g9[7] = fma(w1, dC[1], g9[7]);
                g9[8] = fma(w2, dC[2], g9[8]);
            }
        }
        double g12[12];
#pragma unroll
        for (int k = 0; k < 9; ++k) g12[k] = g9[k];
#pragma unroll
        for (int x = 0; x < 3; ++x) g12[9 + x] = -(g9[x] + g9[3 + x] + g9[6 + x]);
        int idx;
        const double s = warp_sum_transposed<12>(g12, lane, idx);
        if (idx < 12 && (lane & 1) == 0) {
            const int sh = idx < 3 ? q.sa : (idx < 6 ? q.sb : (idx < 9 ? q.sc : q.sd));
            atomicAdd(gshell + 3 * sh + idx % 3, s);
        }
        __syncwarp();   // gam is rewritten for the next item
    }
}

// grad[3 atom] += the atom's shells
__global__ void grad_gather_kernel(int nshell, const int *__restrict__ shell_atom, const double *__restrict__ gshell,
                                   double *grad)
{
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= 3 * nshell) return;
    double s = 0.0;
#pragma unroll 16
    for (int c = 0; c < kGradCopies; ++c) s += gshell[(int64_t)c * 3 * nshell + t];
    atomicAdd(grad + 3 * shell_atom[t / 3] + t % 3, s);
}

cudaError_t launch_grad_gather(int nshell, const int *shell_atom, const double *gshell, double *grad, cudaStream_t st)
{
    if (nshell > 0)
        grad_gather_kernel<<<(3 * nshell + 127) / 128, 128, 0, st>>>(nshell, shell_atom, gshell, grad);
    return cudaGetLastError();
}

// More than 27 components' Gamma and tables leave the registers in thread
// mode; below, a warp's lanes would share too few products.
template <int LA, int LB, int LC, int LD>
static cudaError_t eri_grad_launch(const int4 *list, int nq, const PairInfo *pairs, const PrimPair *prims,
                                   const double *D, double *gshell, int glen, cudaStream_t st, int nsm)
{
    if constexpr (ncart(LA) * ncart(LB) * ncart(LC) * ncart(LD) <= 27) {
        const int grid = grid_blocks(nq, 128, nsm * 32);
        eri_grad_thread_kernel<LA, LB, LC, LD><<<grid, 128, 0, st>>>(list, nq, pairs, prims, D, gshell, glen);
    } else {
        using Lay = GradWarpLayout<LA, LB, LC, LD>;
        auto kern = eri_grad_warp_kernel<LA, LB, LC, LD>;
        const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Lay::bytes);
        if (e != cudaSuccess) return e;
        const int grid = grid_blocks(nq, Lay::warps, nsm * 16);
        kern<<<grid, Lay::warps * 32, Lay::bytes, st>>>(list, nq, pairs, prims, D, gshell, glen);
    }
    return cudaGetLastError();
}

cudaError_t launch_grad(int qc, const int4 *list, int nq, const PairInfo *pairs, const PrimPair *prims,
                        const double *Dscaled, double *gshell, int nshell, cudaStream_t st, int nsm)
{
    if (nq <= 0) return cudaSuccess;
#define PQB_GCASE(CB, CK)                                                                                      \
    case CB *(CB + 1) / 2 + CK:                                                                               \
        return eri_grad_launch<pc_la(CB), pc_lb(CB), pc_la(CK), pc_lb(CK)>(list, nq, pairs, prims, Dscaled, gshell, \
                                                                           3 * nshell, st, nsm);
    switch (qc) {
        PQB_GCASE(0, 0)
        PQB_GCASE(1, 0) PQB_GCASE(1, 1)
        PQB_GCASE(2, 0) PQB_GCASE(2, 1) PQB_GCASE(2, 2)
        PQB_GCASE(3, 0) PQB_GCASE(3, 1) PQB_GCASE(3, 2) PQB_GCASE(3, 3)
        PQB_GCASE(4, 0) PQB_GCASE(4, 1) PQB_GCASE(4, 2) PQB_GCASE(4, 3) PQB_GCASE(4, 4)
        PQB_GCASE(5, 0) PQB_GCASE(5, 1) PQB_GCASE(5, 2) PQB_GCASE(5, 3) PQB_GCASE(5, 4) PQB_GCASE(5, 5)
    default:
        return cudaErrorInvalidValue;
    }
#undef PQB_GCASE
}

}  // namespace pqb
