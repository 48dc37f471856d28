// Coulomb matrix alone (the getJ of a DFT iteration, PyQuante/dft.py:209 and
// :312) in the Hermite Gaussian basis (McMurchie and Davidson, J. Comput. Phys.
// 26, 218 (1978); the density contracted before the integrals: Ahmadi and
// Almlof, Chem. Phys. Lett. 246, 364 (1995)).  With
//   g_a g_b = sum_T E^ab_T Lambda_T   per primitive pair, T = (t,u,v) up to L = La + Lb,
// the integrals never leave the Hermite basis:
//   H^q_U = K_q sum_cd w_cd D_cd E^cd_U                       (hermite_density_kernel)
//   V^p_T = sum_q sum_U (-1)^|U| H^q_U R_(T+U)(p, q) / sqrt(p + q)   (hermite_coulomb_kernel)
//   J_ab  = sum_p K_p sum_T E^ab_T V^p_T                      (hermite_fock_kernel)
// so a primitive quartet costs its Boys function, the R_tuv up to L_p + L_q and
// 2 nherm(L_p) nherm(L_q) multiply-adds: no angular components, no horizontal
// transfer, no digestion, and the pair classes pp and ds are one.
//
// Every unique pair (p, q) is evaluated once and serves both sides.  A thread
// owns a primitive pair p (H^p and V^p in registers) and walks the primitive
// pairs q of a tile, which the block shares; the tile's V^q are sums over the
// warp's lanes, several values at a time by one transposed reduction.
//
// The primitive pairs of each L are sorted by their shell pair's Schwarz factor
// (descending), so the quartets that the plan keeps, Q_ab Q_cd >= threshold,
// are a prefix of the list for every p, and the same quartets are kept here.
#include "eri_engine.cuh"
#include "eri_launch.h"

namespace pqb {

__host__ __device__ constexpr int nherm(int L) { return (L + 1) * (L + 2) * (L + 3) / 6; }
// index of (t, u, v) among all with t + u + v <= L: by order n = t+u+v, then u+v, then v
__host__ __device__ constexpr int herm_index(int t, int u, int v)
{
    const int n = t + u + v, k = u + v;
    return n * (n + 1) * (n + 2) / 6 + k * (k + 1) / 2 + v;
}
__host__ __device__ constexpr int herm_order(int i) { return (i >= 1) + (i >= 4) + (i >= 10) + (i >= 20) + (i >= 35) + (i >= 56) + (i >= 84) + (i >= 120); }
__host__ __device__ constexpr int herm_rest(int i) { return i - herm_order(i) * (herm_order(i) + 1) * (herm_order(i) + 2) / 6; }
__host__ __device__ constexpr int tri_of(int r) { return (r >= 1) + (r >= 3) + (r >= 6) + (r >= 10) + (r >= 15) + (r >= 21) + (r >= 28) + (r >= 36); }
__host__ __device__ constexpr int herm_v(int i) { return herm_rest(i) - tri_of(herm_rest(i)) * (tri_of(herm_rest(i)) + 1) / 2; }
__host__ __device__ constexpr int herm_u(int i) { return tri_of(herm_rest(i)) - herm_v(i); }
__host__ __device__ constexpr int herm_t(int i) { return herm_order(i) - tri_of(herm_rest(i)); }

// E_t of x_A^i x_B^j about P (t <= i + j <= 4), the exponential and K left out
__device__ __forceinline__ void hermite_e(int i, int j, double pa, double pb, double h, double *e)
{
#pragma unroll
    for (int t = 0; t < 5; ++t) e[t] = t == 0 ? 1.0 : 0.0;
    for (int s = 0; s < i + j; ++s) {
        const double d = s < i ? pa : pb;
        double p = 0.0;
#pragma unroll
        for (int t = 0; t < 5; ++t) {
            const double c = e[t];
            e[t] = fma(d, c, fma(h, p, t < 4 ? (t + 1) * e[t + 1 < 5 ? t + 1 : 4] : 0.0));
            p = c;
        }
    }
}

// One thread per primitive pair of the sorted lists: its record.
__global__ void hermite_pairs_kernel(int n, const int2 *__restrict__ src, const PairInfo *__restrict__ pairs,
                                     const PrimPair *__restrict__ prims, const double *__restrict__ Q, JPrim *out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int2 s = src[i];   // pair, primitive pair within it
    const PrimPair &p = prims[pairs[s.x].prim_off + s.y];
    out[i] = JPrim{p.zeta, p.P[0], p.P[1], p.P[2], Q[s.x], s.x, s.y};
}

// One thread per primitive pair: H from the pre-scaled density (both orders of an
// off-diagonal pair).
template <int L>
__global__ void __launch_bounds__(128) hermite_density_kernel(int n, const JPrim *__restrict__ list,
                                                              const PairInfo *__restrict__ pairs,
                                                              const PrimPair *__restrict__ prims,
                                                              const double *__restrict__ D, int nbf, double *__restrict__ H)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const JPrim &q = list[i];
    const PairInfo &pi = pairs[q.pair];
    const PrimPair &p = prims[pi.prim_off + q.prim];
    const double h = 0.5 * p.izeta, w = p.K * (pi.sa == pi.sb ? 1.0 : 2.0);
    double pa[3], pb[3];
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        pa[x] = p.P[x] - pi.A[x];
        pb[x] = pa[x] + pi.AB[x];
    }
    double acc[nherm(L)];
#pragma unroll
    for (int k = 0; k < nherm(L); ++k) acc[k] = 0.0;
    const int na = ncart(pi.la), nb = ncart(pi.lb);
    for (int a = 0; a < na; ++a)
        for (int b = 0; b < nb; ++b) {
            const double d = w * __ldg(D + (int64_t)(pi.fa + a) * nbf + pi.fb + b);
            double ex[5], ey[5], ez[5];
            hermite_e(cart_lx(pi.la, a), cart_lx(pi.lb, b), pa[0], pb[0], h, ex);
            hermite_e(cart_ly(pi.la, a), cart_ly(pi.lb, b), pa[1], pb[1], h, ey);
            hermite_e(cart_lz(pi.la, a), cart_lz(pi.lb, b), pa[2], pb[2], h, ez);
#pragma unroll
            for (int k = 0; k < nherm(L); ++k) acc[k] = fma(d * ex[herm_t(k)], ey[herm_u(k)] * ez[herm_v(k)], acc[k]);
        }
#pragma unroll
    for (int k = 0; k < nherm(L); ++k) H[(int64_t)i * nherm(L) + k] = acc[k];
}

// The same with a warp per primitive pair, for L >= 2: the lanes first make
// the E tables of the three axes (9 powers pairs each), then share the Hermite
// indices.  (A thread's 36 components of a dd pair took 24 us, as long as the
// whole potential of a small molecule.)
template <int L>
__global__ void __launch_bounds__(128) hermite_density_warp_kernel(int n, const JPrim *__restrict__ list,
                                                                   const PairInfo *__restrict__ pairs,
                                                                   const PrimPair *__restrict__ prims,
                                                                   const double *__restrict__ D, int nbf,
                                                                   double *__restrict__ H)
{
    __shared__ double se[4][3][9][5], sd[4][36];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, i = blockIdx.x * 4 + warp;
    if (i >= n) return;   // whole warps
    const JPrim &q = list[i];
    const PairInfo &pi = pairs[q.pair];
    const PrimPair &p = prims[pi.prim_off + q.prim];
    const int la = pi.la, lb = pi.lb, nb = ncart(lb), nab = ncart(la) * nb;
    if (lane < 27) {
        const int x = lane / 9, a = lane % 9 / 3, b = lane % 3;
        const double pa = p.P[x] - pi.A[x];
        double e[5];
        hermite_e(a <= la ? a : 0, b <= lb ? b : 0, pa, pa + pi.AB[x], 0.5 * p.izeta, e);
#pragma unroll
        for (int t = 0; t < 5; ++t) se[warp][x][lane % 9][t] = e[t];
    }
    const double w = p.K * (pi.sa == pi.sb ? 1.0 : 2.0);
    for (int ab = lane; ab < nab; ab += 32)
        sd[warp][ab] = w * __ldg(D + (int64_t)(pi.fa + ab / nb) * nbf + pi.fb + ab % nb);
    __syncwarp();
    for (int k = lane; k < nherm(L); k += 32) {
        const int t = herm_t(k), u = herm_u(k), v = herm_v(k);
        double acc = 0.0;
        for (int a = 0, ab = 0; a < ncart(la); ++a)
            for (int b = 0; b < nb; ++b, ++ab)
                acc = fma(sd[warp][ab] * se[warp][0][3 * cart_lx(la, a) + cart_lx(lb, b)][t],
                          se[warp][1][3 * cart_ly(la, a) + cart_ly(lb, b)][u] *
                              se[warp][2][3 * cart_lz(la, a) + cart_lz(lb, b)][v],
                          acc);
        H[(int64_t)i * nherm(L) + k] = acc;
    }
}

// J of one (pair, component) from the pair's V; first[pair]: its first
// primitive pair in the lists.
__global__ void __launch_bounds__(128) hermite_fock_kernel(int npair, const PairInfo *__restrict__ pairs,
                                                           const PrimPair *__restrict__ prims,
                                                           const int64_t *__restrict__ first, const double *__restrict__ V,
                                                           int nbf, const double *__restrict__ S, double *__restrict__ J)
{
    // a warp per pair: its components, and for each a power-of-two group of
    // lanes that share the primitive pairs
    const int t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (t >= npair) return;   // whole warps
    const PairInfo &pi = pairs[t];
    const int L = pi.la + pi.lb, nh = nherm(L), na = ncart(pi.la), nb = ncart(pi.lb), nab = na * nb;
    const int G = nab == 1 ? 32 : (nab == 3 ? 8 : (nab == 6 ? 4 : (nab == 9 ? 2 : 1))), g = lane & (G - 1);
    const double *v0 = V + first[t];
    for (int c0 = 0; c0 < nab; c0 += 32 / G) {
        const int ab = c0 + lane / G, a = ab / nb, b = ab - a * nb;
        double s = 0.0;
        if (ab < nab) {
            for (int k = g; k < pi.nprim; k += G) {
                const PrimPair &p = prims[pi.prim_off + k];
                const double *v = v0 + (int64_t)k * nh;
                const double h = 0.5 * p.izeta;
                double e[3][5];
#pragma unroll
                for (int x = 0; x < 3; ++x) {
                    const double pa = p.P[x] - pi.A[x];
                    hermite_e(cart_l(pi.la, a, x), cart_l(pi.lb, b, x), pa, pa + pi.AB[x], h, e[x]);
                }
                double r = v[0] * (e[0][0] * e[1][0] * e[2][0]);
                if (L > 0) {   // uniform over the warp
#pragma unroll
                    for (int m = 1; m < nherm(4); ++m)
                        if (m < nh) r = fma(e[0][herm_t(m)] * e[1][herm_u(m)], e[2][herm_v(m)] * v[m], r);
                }
                s = fma(p.K, r, s);
            }
        }
        __syncwarp();
        for (int o = G / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (ab < nab && g == 0) {
            const int64_t i = pi.fa + a, j = pi.fb + b;
            s *= S[i * nbf + j];
            J[i * nbf + j] = s;
            J[j * nbf + i] = s;
        }
    }
}

// F_0 .. F_L for the potential kernels, which are bound by FP64 issue and have
// L1 bandwidth to spare (the reverse of the Fock-build kernels, see boys_os):
// the Taylor coefficients come from the table's rows F_j(T_k) (T_k = k/16, |d|
// <= 1/32, eight terms: below 3e-17 relative) instead of a recursion at T_k, two
// 256-bit loads a lane for L <= 1 (and one of 64 bits for F_1), three above.
//   L <= 1: F_0 and F_1;
//   L = 2 .. 4: F_L and F_(L-1), whose difference gives exp(-T) =
//     (2L-1) F_(L-1) - 2T F_L with an error of an ulp of its terms, all that the
//     downward recursion F_m = (2T F_(m+1) + exp(-T)) / (2m+1) needs;
//   T >= 40: the asymptotic forms of boys_os, evaluated by every lane.
// (0,0) 69 -> 55 FP64 instructions a primitive quartet.
template <int L>
__device__ __forceinline__ void boys_any(double T, double *F)
{
    if constexpr (L > 4) {
        boys<L>(T, F);
    } else {
        constexpr int M0 = L <= 1 ? 0 : L - 1, ROW = L <= 1 ? 8 : 12;   // lowest order of the series; row part read
        const bool big = T >= PQB_BOYS_TMAX;
        const int k = boys_row_index(T * PQB_BOYS_STEP_INV, (int)(PQB_BOYS_TMAX * PQB_BOYS_STEP_INV));
        const double d = fma(k, 1.0 / PQB_BOYS_STEP_INV, -T);
        const double *row = pqb_boys_tab + k * PQB_BOYS_NORD;
        double f[ROW + 1];
#pragma unroll
        for (int j = 0; j < ROW; j += 4) ld4(row + j, f[j], f[j + 1], f[j + 2], f[j + 3]);
        if (L == 1) f[8] = row[8];
        double lo = f[M0 + 7], hi = L >= 1 ? f[M0 + 8] : 0.0;
#pragma unroll
        for (int j = 6; j >= 0; --j) {
            const double dj = d * (1.0 / (j + 1));
            lo = fma(lo, dj, f[M0 + j]);
            if (L >= 1) hi = fma(hi, dj, f[M0 + 1 + j]);
        }
        const double y = rsqrt_nr_unchecked(T);
        if constexpr (L == 0) {
            F[0] = big ? 0.88622692545275801365 * y : lo;
        } else if constexpr (L == 1) {
            const double a0 = 0.88622692545275801365 * y;
            F[0] = big ? a0 : lo;
            F[1] = big ? a0 * (0.5 * y * y) : hi;
        } else {
            const double h = 0.5 * y * y, t2 = 2.0 * T;
            const double e = big ? exp_neg_estimate(T) : fma(-t2, hi, (2 * L - 1) * lo);
            double Ft[L + 1], Fa[L + 1];
            Ft[L] = hi;
            Ft[L - 1] = lo;
#pragma unroll
            for (int m = L - 2; m >= 0; --m) Ft[m] = fma(t2, Ft[m + 1], e) * (1.0 / (2 * m + 1));
            Fa[0] = 0.88622692545275801365 * y;
#pragma unroll
            for (int m = 0; m < L; ++m) Fa[m + 1] = ((2 * m + 1) * Fa[m] - e) * h;
#pragma unroll
            for (int m = 0; m <= L; ++m) F[m] = big ? Fa[m] : Ft[m];
        }
    }
}

// R[herm_index] = R_tuv^(0), t+u+v <= L, from F_m scaled by (-2 alpha)^m: level
// by level, R^(m)_(t+1) = X R^(m+1)_t + t R^(m+1)_(t-1) on the first axis whose
// index is not zero.  R holds, for every tuv, the orders m <= L - (t+u+v) in turn.
template <int L>
__device__ __forceinline__ void hermite_r(const double (&F)[L + 1], double x, double y, double z, double *R)
{
    double lev[L + 1][nherm(L)];   // [m][tuv]; registers, all indices compile-time
#pragma unroll
    for (int m = 0; m <= L; ++m) lev[m][0] = F[m];
#pragma unroll
    for (int i = 1; i < nherm(L); ++i) {
        const int t = herm_t(i), u = herm_u(i), v = herm_v(i);
#pragma unroll
        for (int m = 0; m <= L - herm_order(i); ++m) {
            if (t > 0) {
                const double one = x * lev[m + 1][herm_index(t - 1, u, v)];
                lev[m][i] = t > 1 ? fma((double)(t - 1), lev[m + 1][herm_index(t > 1 ? t - 2 : 0, u, v)], one) : one;
            } else if (u > 0) {
                const double one = y * lev[m + 1][herm_index(t, u - 1, v)];
                lev[m][i] = u > 1 ? fma((double)(u - 1), lev[m + 1][herm_index(t, u > 1 ? u - 2 : 0, v)], one) : one;
            } else {
                const double one = z * lev[m + 1][herm_index(t, u, v - 1)];
                lev[m][i] = v > 1 ? fma((double)(v - 1), lev[m + 1][herm_index(t, u, v > 1 ? v - 2 : 0)], one) : one;
            }
        }
    }
#pragma unroll
    for (int i = 0; i < nherm(L); ++i) R[i] = lev[0][i];
}

// q per reduction batch: the transposed reduction costs about one exchange a
// value from eight values on, and every q of a batch is unrolled code
template <int LQ> struct JBatch {
    static constexpr int NQ = LQ == 0 ? 8 : (LQ == 1 ? 4 : (LQ == 2 ? 2 : 1));
};
constexpr int kJThreads = 128, kJTile = 64;

// V of the lists p (a thread each) and q (kJTile-element tiles of this block's
// chunk) of LP <= LQ: the low momenta are the long lists, which fill the lanes.
// same: one list with itself; then only pairs of q's shell
// pair before p's count for both sides, p's own shell pair for V^p alone.
// Bound by FP64 issue (42-55 % of the FP64 pipe in the eight largest list pairs of
// C8H18 / 6-31G**, N = 210; with s pairs also by the shared-memory wavefronts of
// the tile, 65-79 % of the L1 data pipe): 0.92 ms for the whole matrix, 1.53 ms by
// the Fock-build kernels without exchange.
template <int LP, int LQ>
__global__ void __launch_bounds__(kJThreads) hermite_coulomb_kernel(int np, const JPrim *__restrict__ plist,
                                                                    const double *__restrict__ Hp, double *Vp, int nq,
                                                                    const JPrim *__restrict__ qlist,
                                                                    const double *__restrict__ Hq, double *Vq, int chunk,
                                                                    double thresh)
{
    constexpr bool same = LP == LQ;
    constexpr int NP = nherm(LP), NQH = nherm(LQ), L = LP + LQ, NB = JBatch<LQ>::NQ;
    __shared__ double sq[kJTile][5];        // zeta, P, Q
    __shared__ int spair[kJTile];
    __shared__ double sh[kJTile][NQH];
    const int tid = threadIdx.x, lane = tid & 31, i = blockIdx.x * kJThreads + tid;
    // the grid's second index walks the q list in chunks; a chunk past this
    // block's reach ends at once
    const int q0 = blockIdx.y * chunk, q1 = q0 + chunk < nq ? q0 + chunk : nq;
    const JPrim &head = plist[blockIdx.x * kJThreads];   // the block's largest factor
    if (head.Q * qlist[q0].Q < thresh) return;
    const int last = blockIdx.x * kJThreads + kJThreads - 1 < np ? blockIdx.x * kJThreads + kJThreads - 1 : np - 1;
    if (same && q0 > last && qlist[q0].pair != plist[last].pair) return;
    const bool in = i < np;
    const JPrim p = plist[in ? i : np - 1];
    double h[NP], v[NP];
#pragma unroll
    for (int k = 0; k < NP; ++k) {
        h[k] = in ? Hp[(int64_t)i * NP + k] : 0.0;
        v[k] = 0.0;
    }
    for (int t0 = q0; t0 < q1; t0 += kJTile) {
        // uniform over the block: nothing below the threshold, nothing past this block's shell pairs
        if (head.Q * qlist[t0].Q < thresh) break;
        if (same && t0 > last && qlist[t0].pair != plist[last].pair) break;
        const int nt = q1 - t0 < kJTile ? q1 - t0 : kJTile;
        __syncthreads();
        for (int k = tid; k < nt; k += kJThreads) {
            const JPrim q = qlist[t0 + k];
            sq[k][0] = q.zeta;
            sq[k][1] = q.P[0];
            sq[k][2] = q.P[1];
            sq[k][3] = q.P[2];
            sq[k][4] = q.Q;
            spair[k] = q.pair;
        }
        for (int k = tid; k < nt * NQH; k += kJThreads) (&sh[0][0])[k] = Hq[(int64_t)t0 * NQH + k];
        __syncthreads();
        for (int b0 = 0; b0 < nt; b0 += NB) {
            double part[NB * NQH];
#pragma unroll
            for (int k = 0; k < NB * NQH; ++k) part[k] = 0.0;
            bool any = false;
#pragma unroll
            for (int b = 0; b < NB; ++b) {
                const int k = b0 + b;
                if (k >= nt) break;
                // (t0 + k against i: in one list the order of shell pairs is that of the
                // list, so equal pairs are found by name)
                const bool own = same && spair[k] == p.pair;
                const bool use = in && p.Q * sq[k][4] >= thresh && (!same || own || t0 + k < i);
                if (!__any_sync(0xffffffffu, use)) continue;
                any = true;
                const double x = p.P[0] - sq[k][1], y = p.P[1] - sq[k][2], z = p.P[2] - sq[k][3];
                const double rs = rsqrt_nr_unchecked(p.zeta + sq[k][0]), al = p.zeta * sq[k][0] * rs * rs;
                double F[L + 1], R[nherm(L)];
                boys_any<L>(al * (x * x + y * y + z * z), F);
                double f = use ? rs : 0.0;
#pragma unroll
                for (int m = 0; m <= L; ++m) {
                    F[m] *= f;
                    f *= -2.0 * al;
                }
                hermite_r<L>(F, x, y, z, R);
                const double both = own ? 0.0 : 1.0;
#pragma unroll
                for (int U = 0; U < NQH; ++U) {
                    const double hq = (herm_order(U) & 1) ? -sh[k][U] : sh[k][U];
                    double s = 0.0;
#pragma unroll
                    for (int T = 0; T < NP; ++T) {
                        const double r = R[herm_index(herm_t(T) + herm_t(U), herm_u(T) + herm_u(U), herm_v(T) + herm_v(U))];
                        v[T] = fma(hq, r, v[T]);
                        s = fma(h[T], r, s);
                    }
                    part[b * NQH + U] = same ? s * both : s;
                }
            }
            if (!any) continue;   // uniform over the warp
            // V^q of the batch
#pragma unroll
            for (int r0 = 0; r0 < NB * NQH; r0 += 32) {
                constexpr int K = NB * NQH < 32 ? NB * NQH : 32;
                constexpr int KP = K <= 1 ? 1 : K <= 2 ? 2 : K <= 4 ? 4 : K <= 8 ? 8 : K <= 16 ? 16 : 32;
                double w[K];
#pragma unroll
                for (int k = 0; k < K; ++k) w[k] = r0 + k < NB * NQH ? part[r0 + k < NB * NQH ? r0 + k : 0] : 0.0;
                int idx;
                const double s = warp_sum_transposed<K>(w, lane, idx);
                const int e = r0 + idx, b = e / NQH, U = e - b * NQH;
                if ((lane & (32 / KP - 1)) == 0 && idx < K && e < NB * NQH && b0 + b < nt && s != 0.0)
                    atomicAdd(Vq + (int64_t)(t0 + b0) * NQH + e, (herm_order(U) & 1) ? -s : s);
            }
        }
    }
    if (in) {
#pragma unroll
        for (int k = 0; k < NP; ++k)
            if (v[k] != 0.0) atomicAdd(Vp + (int64_t)i * NP + k, v[k]);
    }
}

// The least chunk of q per block bounds a block's serial chain: the rarer high
// momenta cost up to 3,500 FP64 instructions a primitive quartet.
constexpr int kJLeast[9] = {16, 16, 8, 8, 8, 4, 2, 1, 1};

template <int LP, int LQ>
static cudaError_t launch_coulomb(const JLists &l, double thresh, cudaStream_t st, int nsm)
{
    const int np = l.n[LP], nq = l.n[LQ];
    if (np == 0 || nq == 0) return cudaSuccess;
    // chunks of q: enough blocks for the GPU several times over
    const int bx = (np + kJThreads - 1) / kJThreads;
    int chunk = (int)(((int64_t)nq * bx + nsm * 24 - 1) / (nsm * 24));
    if (chunk < kJLeast[LP + LQ]) chunk = kJLeast[LP + LQ];
    if (chunk > kJTile) chunk = (chunk + kJTile - 1) / kJTile * kJTile;
    hermite_coulomb_kernel<LP, LQ><<<dim3(bx, (nq + chunk - 1) / chunk), kJThreads, 0, st>>>(
        np, l.list + l.off[LP], l.H + l.hoff[LP], l.V + l.hoff[LP], nq, l.list + l.off[LQ], l.H + l.hoff[LQ],
        l.V + l.hoff[LQ], chunk, thresh);
    return cudaGetLastError();
}

cudaError_t launch_hermite_pairs(int n, const int2 *src, const PairInfo *pairs, const PrimPair *prims, const double *Q,
                                 JPrim *out, cudaStream_t st)
{
    if (n > 0) hermite_pairs_kernel<<<(n + 127) / 128, 128, 0, st>>>(n, src, pairs, prims, Q, out);
    return cudaGetLastError();
}

cudaError_t launch_hermite_density(int L, const JLists &l, const PairInfo *pairs, const PrimPair *prims, const double *D,
                                   int nbf, cudaStream_t st)
{
    const int n = l.n[L], grid = (n + 127) / 128;
    if (n == 0) return cudaSuccess;
    const JPrim *list = l.list + l.off[L];
    double *H = l.H + l.hoff[L];
    switch (L) {
    case 0: hermite_density_kernel<0><<<grid, 128, 0, st>>>(n, list, pairs, prims, D, nbf, H); break;
    case 1: hermite_density_kernel<1><<<grid, 128, 0, st>>>(n, list, pairs, prims, D, nbf, H); break;
    case 2: hermite_density_warp_kernel<2><<<(n + 3) / 4, 128, 0, st>>>(n, list, pairs, prims, D, nbf, H); break;
    case 3: hermite_density_warp_kernel<3><<<(n + 3) / 4, 128, 0, st>>>(n, list, pairs, prims, D, nbf, H); break;
    default: hermite_density_warp_kernel<4><<<(n + 3) / 4, 128, 0, st>>>(n, list, pairs, prims, D, nbf, H); break;
    }
    return cudaGetLastError();
}

cudaError_t launch_hermite_coulomb(int LP, int LQ, const JLists &l, double thresh, cudaStream_t st, int nsm)
{
    switch (LQ * (LQ + 1) / 2 + LP) {   // LP <= LQ
    case 0: return launch_coulomb<0, 0>(l, thresh, st, nsm);
    case 1: return launch_coulomb<0, 1>(l, thresh, st, nsm);
    case 2: return launch_coulomb<1, 1>(l, thresh, st, nsm);
    case 3: return launch_coulomb<0, 2>(l, thresh, st, nsm);
    case 4: return launch_coulomb<1, 2>(l, thresh, st, nsm);
    case 5: return launch_coulomb<2, 2>(l, thresh, st, nsm);
    case 6: return launch_coulomb<0, 3>(l, thresh, st, nsm);
    case 7: return launch_coulomb<1, 3>(l, thresh, st, nsm);
    case 8: return launch_coulomb<2, 3>(l, thresh, st, nsm);
    case 9: return launch_coulomb<3, 3>(l, thresh, st, nsm);
    case 10: return launch_coulomb<0, 4>(l, thresh, st, nsm);
    case 11: return launch_coulomb<1, 4>(l, thresh, st, nsm);
    case 12: return launch_coulomb<2, 4>(l, thresh, st, nsm);
    case 13: return launch_coulomb<3, 4>(l, thresh, st, nsm);
    case 14: return launch_coulomb<4, 4>(l, thresh, st, nsm);
    }
    return cudaErrorInvalidValue;
}

cudaError_t launch_hermite_fock(int npair, const PairInfo *pairs, const PrimPair *prims, const int64_t *first,
                                const double *V, int nbf, const double *escale, double *J, cudaStream_t st)
{
    if (npair > 0)
        hermite_fock_kernel<<<(npair + 3) / 4, 128, 0, st>>>(npair, pairs, prims, first, V, nbf, escale, J);
    return cudaGetLastError();
}

}  // namespace pqb
