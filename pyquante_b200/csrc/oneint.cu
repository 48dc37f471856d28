// One-electron integrals (the combinations of Src/cints.c:190-307) and the
// one-electron part of the RHF gradient (PyQuante/force.py:61-64), one warp
// per function pair.
//
// Every one-dimensional factor is a linear form in the moments about A,
//     M_0 = 1, M_1 = PA, M_(k+1) = PA M_k + k/(2g) M_(k-1)     (overlap)
// or in the same moments with the Coulomb kernel's variable u = t^2,
//     G_1 = PA - u PC, G_(k+1) = (PA - u PC) G_k + k (1-u)/(2g) G_(k-1),
// because (x-B)^lj (x-A)^li = sum_p C(lj,p) AB^(lj-p) (x-A)^(li+p); a
// primitive pair whose centre P lies nearer to B takes the moments about B
// instead (the sum would cancel about A).  The binomial coefficients depend on
// the function pair alone: a warp writes both sets to shared memory once.  A
// nuclear-attraction task multiplies the three axes' polynomials in u and pairs
// the product's coefficients with F_m(T), since int_0^1 t^(2m) exp(-T t^2) dt =
// F_m(T): no roots are needed, and the work of a task follows the pair's own
// powers, which are uniform over the warp.
#include <cmath>
#include <cstdint>

#include "oneint.h"
#include "pqb_device.cuh"

namespace pqb {
namespace {

constexpr int kOneWarps = 4;
constexpr int kMaxShell = 3;                       // f functions at most (the host rejects higher ones first)

// Coefficients of (x-A)^li (x-B)^lj in (x-X)^k: about X = A (about = 0)
// C(lj, p) AB^(lj-p) at k = li + p, about X = B C(li, p) (-AB)^(li-p) at
// k = lj + p; 0 elsewhere.
__device__ double moment_coef(int about, int li, int lj, int k, double ab)
{
    if (about) {
        const int l = li;
        li = lj;
        lj = l;
        ab = -ab;
    }
    const int p = k - li;
    if (li < 0 || lj < 0 || p < 0 || p > lj) return 0.0;
    double r = 1.0;
    for (int q = 1; q <= p; ++q) r = r * (lj - p + q) / q;
    for (int q = p; q < lj; ++q) r *= ab;
    return r;
}

__device__ __forceinline__ void pair_of_index(int64_t t, int &i, int &j)
{
    i = (int)((sqrt(8.0 * (double)t + 1.0) - 1.0) * 0.5);
    while ((int64_t)i * (i + 1) / 2 > t) --i;
    while ((int64_t)(i + 1) * (i + 2) / 2 <= t) ++i;
    j = (int)(t - (int64_t)i * (i + 1) / 2);
}

__device__ __forceinline__ double warp_total(double x)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

template <int L>
__device__ __forceinline__ void boys_upto(double T, double *F)
{
    if constexpr (L <= 4)
        boys_os<L>(T, F);
    else
        boys<L>(T, F);
}

// r[0..D] = NV linear forms (coefficients cv[v][k], k <= nb <= D) of the
// polynomials G_0 .. G_nb in u of one axis; nb is uniform over the warp.
template <int D, int NV>
__device__ __forceinline__ void axis_poly(double pa, double pc, double o2g, int nb, const double *cv, int stride,
                                          double (*r)[D + 1])
{
    double gp[D + 1], g[D + 1];
#pragma unroll
    for (int d = 0; d <= D; ++d) gp[d] = g[d] = 0.0;
    g[0] = 1.0;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
#pragma unroll
        for (int d = 0; d <= D; ++d) r[v][d] = 0.0;
        r[v][0] = cv[v * stride];
    }
#pragma unroll
    for (int k = 0; k < D; ++k) {
        if (k < nb) {
            const double b = k * o2g;
            double gn[D + 1];
#pragma unroll
            for (int d = 0; d <= k + 1; ++d) {
                double t = d <= k ? pa * g[d] : 0.0;
                if (d > 0) t = fma(-pc, g[d - 1], t);
                if (k > 0) {
                    if (d <= k - 1) t = fma(b, gp[d], t);
                    if (d > 0) t = fma(-b, gp[d - 1], t);
                }
                gn[d] = t;
            }
#pragma unroll
            for (int d = 0; d <= k; ++d) gp[d] = g[d];
#pragma unroll
            for (int d = 0; d <= k + 1; ++d) g[d] = gn[d];
#pragma unroll
            for (int v = 0; v < NV; ++v) {
                const double c = cv[v * stride + k + 1];
#pragma unroll
                for (int d = 0; d <= k + 1; ++d) r[v][d] = fma(c, gn[d], r[v][d]);
            }
        }
    }
}

// x <- x y in u, degrees adding up to at most D (so nothing is cut off)
template <int D>
__device__ __forceinline__ void poly_mul(double *x, const double *y)
{
#pragma unroll
    for (int d = D; d >= 0; --d) {
        double t = x[d] * y[0];
#pragma unroll
        for (int k = 1; k <= d; ++k) t = fma(x[d - k], y[k], t);
        x[d] = t;
    }
}

// the primitive pairs of one chunk that survive their Gaussian factor
struct OnePrims {
    double P[3][32], g[32], o2g[32], pre[32];
    int about[32];         // 0: moments about A, 1: about B
};

struct OneWarp {
    double cv[2][3][3][10];   // [about][axis][lj - 2, lj, lj + 2][k <= 8]
    OnePrims pp;
};

// -sum_C Z_C <i|1/|r-C||j> over the chunk's primitive pairs and all atoms;
// the lanes share the np x natoms tasks.
template <int L>
__device__ __forceinline__ double attraction(const OneWarp &w, const double *A, const double *AB, const int *nb,
                                             int np, int natoms, const double *__restrict__ atoms, int lane)
{
    double sum = 0.0;
    const int stepp = 32 / natoms, stepc = 32 - stepp * natoms;
    int p = lane / natoms, c = lane - (lane / natoms) * natoms;
    while (p < np) {
        double Cx, Cy, Cz, Z;
        ld4(atoms + 4 * c, Cx, Cy, Cz, Z);
        const double g = w.pp.g[p], o2g = w.pp.o2g[p];
        const double P[3] = {w.pp.P[0][p], w.pp.P[1][p], w.pp.P[2][p]};
        const double PC[3] = {P[0] - Cx, P[1] - Cy, P[2] - Cz};
        double F[L + 1];
        boys_upto<L>(g * (PC[0] * PC[0] + PC[1] * PC[1] + PC[2] * PC[2]), F);
        double q[L + 1];
#pragma unroll
        for (int d = 0; d <= L; ++d) q[d] = 0.0;
        q[0] = 1.0;
        if constexpr (L > 0) {
            const int ab = w.pp.about[p];
#pragma unroll
            for (int x = 0; x < 3; ++x)
                if (nb[x] > 0) {
                    double r[1][L + 1];
                    axis_poly<L, 1>(P[x] - (ab ? A[x] - AB[x] : A[x]), PC[x], o2g, nb[x], w.cv[ab][x][1], 0, r);
                    poly_mul<L>(q, r[0]);
                }
        }
        double acc = q[0] * F[0];
#pragma unroll
        for (int d = 1; d <= L; ++d) acc = fma(q[d], F[d], acc);
        sum = fma(-Z * w.pp.pre[p], acc, sum);
        p += stepp;
        c += stepc;
        if (c >= natoms) {
            c -= natoms;
            ++p;
        }
    }
    return sum;
}

// One warp per pair i >= j, S, T and V being symmetric.  A chunk of 32
// primitive pairs goes first, one per lane (overlap and kinetic terms there,
// the pair's data to shared memory unless its Gaussian factor is exactly
// zero); then the lanes share the chunk's (primitive pair, atom) tasks.
// Bound by FP64 latency and issue: C16H34 / 6-31G* (N = 308, 50 atoms) takes
// 0.24 ms (0.27 with the registers uncapped, 12 warps an SM instead of 20); 11.6
// ms with one thread per (i, j), which looped over its primitives, atoms and Rys
// roots in local-memory tables, the lanes of a warp on unlike powers.
__global__ void __launch_bounds__(kOneWarps * 32, 5) oneint_kernel(int n, FuncTable ft, int natoms,
                                                                const double *__restrict__ atoms, double *S,
                                                                double *Tk, double *V)
{
    __shared__ OneWarp sw[kOneWarps];
    const int lane = threadIdx.x & 31;
    OneWarp &w = sw[threadIdx.x >> 5];
    const int64_t t = (int64_t)blockIdx.x * kOneWarps + (threadIdx.x >> 5);
    if (t >= (int64_t)n * (n + 1) / 2) return;   // whole warps
    int i, j;
    pair_of_index(t, i, j);
    double A[3], AB[3], rab2 = 0.0;
    int li[3], lj[3], nb[3], Li = 0, Lj = 0;
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        A[x] = ft.origin[3 * i + x];
        AB[x] = A[x] - ft.origin[3 * j + x];
        rab2 += AB[x] * AB[x];
        li[x] = ft.powers[3 * i + x];
        lj[x] = ft.powers[3 * j + x];
        nb[x] = li[x] + lj[x];
        Li += li[x];
        Lj += lj[x];
    }
    double s_sum = 0.0, t_sum = 0.0, v_sum = 0.0;
    if (Li > kMaxShell || Lj > kMaxShell) {
        s_sum = t_sum = v_sum = nan("");
    } else {
        for (int e = lane; e < 2 * 3 * 3 * 9; e += 32) {
            const int s = e / 81, x = (e - s * 81) / 27, v = (e % 27) / 9, k = e % 9;
            w.cv[s][x][v][k] = moment_coef(s, li[x], lj[x] + 2 * v - 2, k, AB[x]);
        }
        __syncwarp();
        const int pi0 = ft.prim_off[i], ni = ft.prim_off[i + 1] - pi0, pj0 = ft.prim_off[j],
                  nj = ft.prim_off[j + 1] - pj0;
        for (int c0 = 0; c0 < ni * nj; c0 += 32) {
            const int pq = c0 + lane;
            bool keep = pq < ni * nj;
            double g = 1.0, pre = 0.0, P[3] = {0.0, 0.0, 0.0}, o2g = 0.5;
            int ab = 0;
            if (keep) {
                const int p = pq / nj, q = pq - p * nj;
                const double a = ft.exps[pi0 + p], b = ft.exps[pj0 + q];
                g = a + b;
                ab = b > a;
                const double ig = 1.0 / g;
                o2g = 0.5 * ig;
                const double Ew = exp(-a * b * ig * rab2) * ft.cn[pi0 + p] * ft.cn[pj0 + q];
                pre = 2.0 * kPi * ig * Ew;
                keep = Ew != 0.0;
                // one-dimensional overlaps with lj - 2, lj, lj + 2
                double s[3][3];
#pragma unroll
                for (int x = 0; x < 3; ++x) {
                    // P - A = -(b/g) AB, P - B = (a/g) AB: no cancellation
                    const double px = (ab ? a : -b) * ig * AB[x];
                    P[x] = (ab ? A[x] - AB[x] : A[x]) + px;
                    const double (*cv)[10] = w.cv[ab][x];
                    double mp = 0.0, m = 1.0;
#pragma unroll
                    for (int v = 0; v < 3; ++v) s[x][v] = cv[v][0];
                    for (int k = 0; k < nb[x] + 2; ++k) {
                        const double mn = fma(px, m, k * o2g * mp);
                        mp = m;
                        m = mn;
#pragma unroll
                        for (int v = 0; v < 3; ++v) s[x][v] = fma(cv[v][k + 1], m, s[x][v]);
                    }
                }
                const double pis = kPi * ig, ov = pis * sqrt(pis) * Ew;
                double tk = 0.0;
#pragma unroll
                for (int x = 0; x < 3; ++x) {
                    const int l = lj[x];
                    const double tx = b * (2 * l + 1) * s[x][1] - 2.0 * b * b * s[x][2] - 0.5 * l * (l - 1) * s[x][0];
                    tk = fma(tx * s[(x + 1) % 3][1], s[(x + 2) % 3][1], tk);
                }
                s_sum = fma(ov, s[0][1] * s[1][1] * s[2][1], s_sum);
                t_sum = fma(ov, tk, t_sum);
            }
            if (V && natoms > 0) {   // uniform over the grid
                const unsigned m = __ballot_sync(0xffffffffu, keep);
                const int np = __popc(m);
                if (keep) {
                    const int at = __popc(m & ((1u << lane) - 1u));
#pragma unroll
                    for (int x = 0; x < 3; ++x) w.pp.P[x][at] = P[x];
                    w.pp.g[at] = g;
                    w.pp.o2g[at] = o2g;
                    w.pp.pre[at] = pre;
                    w.pp.about[at] = ab;
                }
                __syncwarp();
                switch (Li + Lj) {   // uniform over the warp
                case 0: v_sum += attraction<0>(w, A, AB, nb, np, natoms, atoms, lane); break;
                case 1: v_sum += attraction<1>(w, A, AB, nb, np, natoms, atoms, lane); break;
                case 2: v_sum += attraction<2>(w, A, AB, nb, np, natoms, atoms, lane); break;
                case 3: v_sum += attraction<3>(w, A, AB, nb, np, natoms, atoms, lane); break;
                case 4: v_sum += attraction<4>(w, A, AB, nb, np, natoms, atoms, lane); break;
                case 5: v_sum += attraction<5>(w, A, AB, nb, np, natoms, atoms, lane); break;
                default: v_sum += attraction<6>(w, A, AB, nb, np, natoms, atoms, lane); break;
                }
                __syncwarp();   // the next chunk overwrites the shared pairs
            }
        }
    }
    s_sum = warp_total(s_sum);
    t_sum = warp_total(t_sum);
    v_sum = warp_total(v_sum);
    if (lane == 0) {
        const double nn = ft.norms[i] * ft.norms[j];
        const int64_t ij = (int64_t)i * n + j, ji = (int64_t)j * n + i;
        if (S) S[ij] = S[ji] = nn * s_sum;
        if (Tk) Tk[ij] = Tk[ji] = nn * t_sum;
        if (V) V[ij] = V[ji] = nn * v_sum;
    }
}

// ---- gradient -----------------------------------------------------------
// d/dA_x g_a = 2 alpha g_(a+1x) - a_x g_(a-1x); dS/dB = -dS/dA, dT/dB =
// -dT/dA; for each nucleus C the Hellmann-Feynman term
// dV_C/dC = -(dV_C/dA + dV_C/dB).
struct GradWarp {
    double cv[2][3][3][3][11];   // [about][axis][li - 1, li, li + 1][lj - 2, lj, lj + 2][k <= 9]
    double cb[2][3][2][11];      // [about][axis] (li, lj - 1), (li, lj + 1)
    OnePrims pp;
    double a2[32], b2[32];    // 2 alpha, 2 beta
};

// The attraction's derivatives of one (primitive pair, atom): vA, vB without
// the prefactor.  D = Li + Lj + 1.
template <int D>
__device__ __forceinline__ void attraction_grad(const GradWarp &w, int p, const double *A, const double *AB,
                                                const int *li, const int *lj, double Cx, double Cy, double Cz,
                                                double *vA, double *vB)
{
    const double g = w.pp.g[p], o2g = w.pp.o2g[p], a2 = w.a2[p], b2 = w.b2[p];
    const double P[3] = {w.pp.P[0][p], w.pp.P[1][p], w.pp.P[2][p]};
    const double PC[3] = {P[0] - Cx, P[1] - Cy, P[2] - Cz};
    double F[D + 1];
    boys_upto<D>(g * (PC[0] * PC[0] + PC[1] * PC[1] + PC[2] * PC[2]), F);
    double I0[3][D + 1], IA[3][D + 1], IB[3][D + 1];
    const int ab = w.pp.about[p];
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        const int nb = li[x] + lj[x] + 1;
        const double px = P[x] - (ab ? A[x] - AB[x] : A[x]);
        // (li - 1, lj), (li, lj), (li + 1, lj) at a stride of 3 x 11; (li, lj - 1), (li, lj + 1)
        double r[3][D + 1], rb[2][D + 1];
        axis_poly<D, 3>(px, PC[x], o2g, nb, w.cv[ab][x][0][1], 33, r);
        axis_poly<D, 2>(px, PC[x], o2g, nb, w.cb[ab][x][0], 11, rb);
        const double l = li[x], m = lj[x];
#pragma unroll
        for (int d = 0; d <= D; ++d) {
            I0[x][d] = r[1][d];
            IA[x][d] = a2 * r[2][d] - l * r[0][d];
            IB[x][d] = b2 * rb[1][d] - m * rb[0][d];
        }
    }
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        const int y = (x + 1) % 3, z = (x + 2) % 3;
        double q[D + 1];
#pragma unroll
        for (int d = 0; d <= D; ++d) q[d] = I0[y][d];
        poly_mul<D>(q, I0[z]);
        double sa = 0.0, sb = 0.0;
#pragma unroll
        for (int d = 0; d <= D; ++d) {
            double f = 0.0;
#pragma unroll
            for (int e = 0; e + d <= D; ++e) f = fma(q[e], F[e + d], f);
            sa = fma(IA[x][d], f, sa);
            sb = fma(IB[x][d], f, sb);
        }
        vA[x] = sa;
        vB[x] = sb;
    }
}

// Lanes = atoms (a power-of-two group G >= natoms of lanes, 32 / G primitive
// pairs side by side; natoms > 32: one atom block after the other), so a
// nucleus's term is summed in registers over the primitive pairs.  gout:
// where this warp adds its gradient (its own shared array, or global memory
// by atomics for more than kGradSharedAtoms atoms).
constexpr int kGradSharedAtoms = 128;

template <int D>
__device__ __forceinline__ void attraction_grad_all(const GradWarp &w, const double *A, const double *AB,
                                                    const int *li, const int *lj, int np, int natoms,
                                                    const double *__restrict__ atoms, double d2, int lane,
                                                    double *gA, double *gB, double *gs, double *grad)
{
    int G = 1;
    while (G < 32 && G < natoms) G <<= 1;
    const int sub = lane / G, la = lane & (G - 1);
    for (int c0 = 0; c0 < natoms; c0 += G) {
        const int c = c0 + la;
        double gC[3] = {0.0, 0.0, 0.0};
        if (c < natoms) {
            double Cx, Cy, Cz, Z;
            ld4(atoms + 4 * c, Cx, Cy, Cz, Z);
            for (int p = sub; p < np; p += 32 / G) {
                double vA[3], vB[3];
                attraction_grad<D>(w, p, A, AB, li, lj, Cx, Cy, Cz, vA, vB);
                const double zf = -Z * w.pp.pre[p] * d2;
#pragma unroll
                for (int x = 0; x < 3; ++x) {
                    gA[x] = fma(zf, vA[x], gA[x]);
                    gB[x] = fma(zf, vB[x], gB[x]);
                    gC[x] = fma(-zf, vA[x] + vB[x], gC[x]);
                }
            }
        }
        __syncwarp();
#pragma unroll
        for (int x = 0; x < 3; ++x)
            for (int o = 16; o >= G; o >>= 1) gC[x] += __shfl_xor_sync(0xffffffffu, gC[x], o);
        if (sub == 0 && c < natoms) {
#pragma unroll
            for (int x = 0; x < 3; ++x) {
                if (gs)
                    gs[3 * c + x] += gC[x];
                else
                    atomicAdd(grad + 3 * c + x, gC[x]);
            }
        }
    }
}

// One warp per pair i >= j (weights of both orders), pairs strided over the
// warps of a resident grid so that the nuclei's terms stay in shared memory
// until the block's end.  (H2O)4 / 6-31G* (N = 76) took 9.2 ms with one
// thread per (i, j) and three global atomics per (primitive pair, nucleus).
__global__ void __launch_bounds__(kOneWarps * 32) oneint_grad_kernel(int n, FuncTable ft, int natoms,
                                                                     const double *__restrict__ atoms,
                                                                     const int *__restrict__ func_atom,
                                                                     const double *__restrict__ Dm,
                                                                     const double *__restrict__ Wm, double *grad)
{
    __shared__ GradWarp sw[kOneWarps];
    extern __shared__ double sg[];   // [warp][3 natoms], natoms <= kGradSharedAtoms
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    GradWarp &w = sw[warp];
    const bool shared = natoms <= kGradSharedAtoms;
    double *gs = shared ? sg + warp * 3 * natoms : nullptr;
    if (shared)
        for (int e = lane; e < 3 * natoms; e += 32) gs[e] = 0.0;
    __syncwarp();
    const int64_t npairs = (int64_t)n * (n + 1) / 2;
    for (int64_t t = (int64_t)blockIdx.x * kOneWarps + warp; t < npairs; t += (int64_t)gridDim.x * kOneWarps) {
        int i, j;
        pair_of_index(t, i, j);
        double A[3], AB[3], rab2 = 0.0;
        int li[3], lj[3], Li = 0, Lj = 0;
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            A[x] = ft.origin[3 * i + x];
            AB[x] = A[x] - ft.origin[3 * j + x];
            rab2 += AB[x] * AB[x];
            li[x] = ft.powers[3 * i + x];
            lj[x] = ft.powers[3 * j + x];
            Li += li[x];
            Lj += lj[x];
        }
        if (Li > kMaxShell || Lj > kMaxShell) continue;   // the host rejects these first
        const int64_t ij = (int64_t)i * n + j, ji = (int64_t)j * n + i;
        const double nn = 2.0 * ft.norms[i] * ft.norms[j];
        const double d2 = nn * (i == j ? Dm[ij] : Dm[ij] + Dm[ji]), w2 = nn * (i == j ? Wm[ij] : Wm[ij] + Wm[ji]);
        __syncwarp();
        for (int e = lane; e < 2 * 3 * 9 * 10; e += 32) {
            const int s = e / 270, x = (e % 270) / 90, u = (e % 90) / 30, v = (e % 30) / 10, k = e % 10;
            w.cv[s][x][u][v][k] = moment_coef(s, li[x] + u - 1, lj[x] + 2 * v - 2, k, AB[x]);
        }
        for (int e = lane; e < 2 * 3 * 2 * 10; e += 32) {
            const int s = e / 60, x = (e % 60) / 20, v = (e % 20) / 10, k = e % 10;
            w.cb[s][x][v][k] = moment_coef(s, li[x], lj[x] + 2 * v - 1, k, AB[x]);
        }
        __syncwarp();
        double gA[3] = {0.0, 0.0, 0.0}, gB[3] = {0.0, 0.0, 0.0};
        const int pi0 = ft.prim_off[i], ni = ft.prim_off[i + 1] - pi0, pj0 = ft.prim_off[j],
                  nj = ft.prim_off[j + 1] - pj0;
        for (int c0 = 0; c0 < ni * nj; c0 += 32) {
            const int pq = c0 + lane;
            bool keep = pq < ni * nj;
            double a = 1.0, b = 1.0, g = 2.0, o2g = 0.25, pre = 0.0, P[3] = {0.0, 0.0, 0.0};
            int ab = 0;
            if (keep) {
                const int p = pq / nj, q = pq - p * nj;
                a = ft.exps[pi0 + p];
                b = ft.exps[pj0 + q];
                g = a + b;
                ab = b > a;
                const double ig = 1.0 / g;
                o2g = 0.5 * ig;
                const double Ew = exp(-a * b * ig * rab2) * ft.cn[pi0 + p] * ft.cn[pj0 + q];
                pre = 2.0 * kPi * ig * Ew;
                keep = Ew != 0.0;
                double S0[3], dS[3], T0[3], dT[3];
#pragma unroll
                for (int x = 0; x < 3; ++x) {
                    const double px = (ab ? a : -b) * ig * AB[x];
                    P[x] = (ab ? A[x] - AB[x] : A[x]) + px;
                    const double (*cv)[3][11] = w.cv[ab][x];
                    double s[3][3], mp = 0.0, m = 1.0;
#pragma unroll
                    for (int u = 0; u < 3; ++u)
#pragma unroll
                        for (int v = 0; v < 3; ++v) s[u][v] = cv[u][v][0];
                    for (int k = 0; k < li[x] + lj[x] + 3; ++k) {
                        const double mn = fma(px, m, k * o2g * mp);
                        mp = m;
                        m = mn;
#pragma unroll
                        for (int u = 0; u < 3; ++u)
#pragma unroll
                            for (int v = 0; v < 3; ++v) s[u][v] = fma(cv[u][v][k + 1], m, s[u][v]);
                    }
                    const int l = lj[x];
                    double kin[3];
#pragma unroll
                    for (int u = 0; u < 3; ++u)
                        kin[u] = b * (2 * l + 1) * s[u][1] - 2.0 * b * b * s[u][2] - 0.5 * l * (l - 1) * s[u][0];
                    S0[x] = s[1][1];
                    T0[x] = kin[1];
                    dS[x] = 2.0 * a * s[2][1] - li[x] * s[0][1];
                    dT[x] = 2.0 * a * kin[2] - li[x] * kin[0];
                }
                const double pis = kPi * ig, ov = pis * sqrt(pis) * Ew;
#pragma unroll
                for (int x = 0; x < 3; ++x) {
                    const int y = (x + 1) % 3, z = (x + 2) % 3;
                    const double ds = dS[x] * S0[y] * S0[z];
                    const double dt = dT[x] * S0[y] * S0[z] + dS[x] * (T0[y] * S0[z] + S0[y] * T0[z]);
                    const double c = ov * (d2 * dt - w2 * ds);
                    gA[x] += c;
                    gB[x] -= c;
                }
            }
            const unsigned m = __ballot_sync(0xffffffffu, keep);
            const int np = __popc(m);
            if (keep) {
                const int at = __popc(m & ((1u << lane) - 1u));
#pragma unroll
                for (int x = 0; x < 3; ++x) w.pp.P[x][at] = P[x];
                w.pp.g[at] = g;
                w.pp.o2g[at] = o2g;
                w.pp.pre[at] = pre;
                w.pp.about[at] = ab;
                w.a2[at] = 2.0 * a;
                w.b2[at] = 2.0 * b;
            }
            __syncwarp();
            switch (Li + Lj) {   // uniform over the warp
            case 0: attraction_grad_all<1>(w, A, AB, li, lj, np, natoms, atoms, d2, lane, gA, gB, gs, grad); break;
            case 1: attraction_grad_all<2>(w, A, AB, li, lj, np, natoms, atoms, d2, lane, gA, gB, gs, grad); break;
            case 2: attraction_grad_all<3>(w, A, AB, li, lj, np, natoms, atoms, d2, lane, gA, gB, gs, grad); break;
            case 3: attraction_grad_all<4>(w, A, AB, li, lj, np, natoms, atoms, d2, lane, gA, gB, gs, grad); break;
            case 4: attraction_grad_all<5>(w, A, AB, li, lj, np, natoms, atoms, d2, lane, gA, gB, gs, grad); break;
            case 5: attraction_grad_all<6>(w, A, AB, li, lj, np, natoms, atoms, d2, lane, gA, gB, gs, grad); break;
            default: attraction_grad_all<7>(w, A, AB, li, lj, np, natoms, atoms, d2, lane, gA, gB, gs, grad); break;
            }
            __syncwarp();
        }
        const int ai = func_atom[i], aj = func_atom[j];
#pragma unroll
        for (int x = 0; x < 3; ++x) {
            const double ga = warp_total(gA[x]), gb = warp_total(gB[x]);
            if (lane == 0) {
                if (gs) {
                    gs[3 * ai + x] += ga;
                    gs[3 * aj + x] += gb;
                } else {
                    atomicAdd(grad + 3 * ai + x, ga);
                    atomicAdd(grad + 3 * aj + x, gb);
                }
            }
        }
        __syncwarp();
    }
    if (shared) {
        __syncthreads();
        for (int e = threadIdx.x; e < 3 * natoms; e += kOneWarps * 32) {
            double s = 0.0;
#pragma unroll
            for (int v = 0; v < kOneWarps; ++v) s += sg[v * 3 * natoms + e];
            if (s != 0.0) atomicAdd(grad + e, s);
        }
    }
}

}  // namespace

cudaError_t launch_oneint_grad(int n, const FuncTable &ft, int natoms, const double *atoms, const int *func_atom,
                               const double *D, const double *W, double *grad, cudaStream_t st, int nsm)
{
    const int64_t pairs = (int64_t)n * (n + 1) / 2, blocks = (pairs + kOneWarps - 1) / kOneWarps;
    const size_t smem = natoms <= kGradSharedAtoms ? sizeof(double) * kOneWarps * 3 * natoms : 0;
    // two resident blocks per SM by registers
    const int grid = (int)(blocks < 2 * nsm ? blocks : 2 * nsm);
    oneint_grad_kernel<<<grid, kOneWarps * 32, smem, st>>>(n, ft, natoms, atoms, func_atom, D, W, grad);
    return cudaGetLastError();
}

cudaError_t launch_oneint(int n, const FuncTable &ft, int natoms, const double *atoms, double *S, double *Tk, double *V,
                          cudaStream_t st)
{
    const int64_t pairs = (int64_t)n * (n + 1) / 2;
    oneint_kernel<<<(unsigned)((pairs + kOneWarps - 1) / kOneWarps), kOneWarps * 32, 0, st>>>(n, ft, natoms, atoms, S,
                                                                                              Tk, V);
    return cudaGetLastError();
}

}  // namespace pqb
