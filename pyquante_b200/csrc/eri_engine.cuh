// Shell-quartet ERI engine: one kernel template per angular-momentum class
// (LA LB | LC LD), fed a class-sorted list of (bra pair, ket pair) quartets.
//
// Two integral schemes, chosen per class at compile time:
//  * classes with LA+LB+LC+LD <= 4 (thread mode): the Obara--Saika vertical
//    recurrence per primitive quartet and the Head-Gordon--Pople horizontal
//    transfer once per contracted item (the scheme of the reference's
//    Src/chgp.c:78-419), as straight-line code generated by gen_os.py
//    (os_classes.inc);
//  * the rest: the Rys quadrature of the reference's Src/crys.c:56-97 (sum
//    over roots of Ix*Iy*Iz*w, ABD eqs 5, 9).
// Both are organised per SHELL quartet: the recurrences run once per
// primitive quartet and serve every cartesian component, instead of once per
// component as crys.contr_coulomb does (Src/crys.c:34-54).
//
// Two execution modes:
//  * thread mode (NAB*NCD <= 81, which is every class with L <= 4): one
//    thread per work item; the recurrence intermediates and all contracted
//    components live in registers.
//  * warp mode (larger classes, FP64 in both precision modes): a warp holds
//    32/NCD quartets, a lane per ket component pair; per primitive quartet the
//    lanes share the roots and the 2-D integrals, which go to shared memory,
//    then every lane accumulates the NAB bra components of its ket component
//    pair in registers.
//
// The epilogue functor consumes a quartet's contracted integrals (thread
// mode) or those of one ket component pair (warp mode), so the same engine
// writes packed integrals, digests into J/K, or forms Schwarz bounds.
#pragma once
#include <atomic>
#include <type_traits>
#include "pqb_device.cuh"
#include "pqb_types.h"

namespace pqb {

struct QCtx {
    int fa, fb, fc, fd;   // first function index of the four shells
    int sa, sb, sc, sd;   // shell indices
    int bra, ket;         // pair ids (bra == ket: diagonal quartet)
    int nm;               // row length of the molecule's D/J/K block
    long long bo;         // element (i, j) of that block: bo + i*nm + j
};

__device__ __forceinline__ QCtx make_qctx(const PairInfo &pb, const PairInfo &pk, int bra, int ket)
{
    return QCtx{pb.fa, pb.fb, pk.fa, pk.fb, pb.sa, pb.sb, pk.sa, pk.sb, bra, ket, pb.nm, pb.bo};
}

__device__ __forceinline__ int64_t fpair(int i, int j)
{
    return i >= j ? (int64_t)i * (i + 1) / 2 + j : (int64_t)j * (j + 1) / 2 + i;
}

// ------------------------------------------------------------ epilogues --
// Every epilogue offers
//   thread_quartet<LA,LB,LC,LD>(q, acc[NAB*NCD], lane, live)
//                                                  whole quartet, thread mode (all lanes
//                                                  of the warp call it; live = a real item)
//   lane_quartet<LA,LB,LC,LD>(q, ic, id, lane, live, acc[NAB], buf)
//                                                  one ket component pair of a quartet,
//                                                  warp mode (all lanes of the warp call it)

// 1 if (x0, y0) > (x1, y1) lexicographically, 1/2 if equal, 0 if less.
__host__ __device__ constexpr double lex_weight(int x0, int y0, int x1, int y1)
{
    return x0 != x1 ? (x0 > x1 ? 1.0 : 0.0) : (y0 != y1 ? (y0 > y1 ? 1.0 : 0.0) : 0.5);
}

// Degeneracy weight of component (ia ib|ic id) of a unique shell quartet:
// 0 outside the canonical ranges i >= j, k >= l, ij >= kl; a factor 1/2 for
// each of i == j, k == l, ij == kl; else 1.  Only the flags are runtime:
//   bd: the bra's two shells are one shell (then i - j = ia - ib),
//   kd: the same for the ket,
//   qd: bra pair == ket pair (then IJ vs KL orders (ia, ib) vs (ic, id)
//       lexicographically when the first shell holds the higher function
//       indices, af, or bd; otherwise (ib, ia) vs (id, ic)).
// In the unrolled loops the component indices are constants, so each weight
// is a few selects: no branches and no 64-bit pair indices per component.
__device__ __forceinline__ double comp_weight(int ia, int ib, int ic, int id, bool bd, bool kd, bool qd, bool af)
{
    const double wb = ia > ib ? 1.0 : (ia == ib ? 0.5 : 0.0);
    const double wk = ic > id ? 1.0 : (ic == id ? 0.5 : 0.0);
    const double wq = (bd || af) ? lex_weight(ia, ib, ic, id) : lex_weight(ib, ia, id, ic);
    return (bd ? wb : 1.0) * (kd ? wk : 1.0) * (qd ? wq : 1.0);
}

// Packed canonical integrals at ijkl2intindex (Src/cints.c:413-425), 64-bit.
// Bound by the L2's rate of partial-sector writes (about 105 G sectors/s;
// a row's neighbouring elements come from other classes' quartets, so a thread
// owns only the run of consecutive elements that one shell gives): runs go out
// 16 bytes at a time.  Which index runs is decided per quartet by the shells'
// order, so the component loops hold no comparisons.  (H2O)6 / 6-31G** (N = 150,
// 513 MB): 1.36 -> 1.01 ms a call, 107 -> 86 M sectors; the kernels one after the
// other 2.20 -> 1.37 ms, of which the sharing of long items (kCoopLanes) took
// (00|00), with items of 1,296 primitive quartets, from 0.34 to 0.08.
struct EpiPacked {
    double *out;
    const double *fscale;
    static constexpr bool kCoop = true;
    __device__ __forceinline__ bool screened(const PairInfo &, const PairInfo &, int, int) const { return false; }

    // p[n] = x[n S] f[n] s, n < N, f the component scales of functions f0 ..
    template <int N, int S, typename R>
    __device__ __forceinline__ void run(double *p, const R *x, int f0, double s) const
    {
        double v[N];
#pragma unroll
        for (int n = 0; n < N; ++n) v[n] = (double)x[n * S] * (s * __ldg(fscale + f0 + n));
        if constexpr (N == 1) {
            p[0] = v[0];
        } else if (reinterpret_cast<uintptr_t>(p) & 8) {
            p[0] = v[0];
#pragma unroll
            for (int n = 1; n + 1 < N; n += 2) *reinterpret_cast<double2 *>(p + n) = make_double2(v[n], v[n + 1]);
            if (N % 2 == 0) p[N - 1] = v[N - 1];
        } else {
#pragma unroll
            for (int n = 0; n + 1 < N; n += 2) *reinterpret_cast<double2 *>(p + n) = make_double2(v[n], v[n + 1]);
            if (N % 2 == 1) p[N - 1] = v[N - 1];
        }
    }
    // the row of the packed array that starts at (IJ|0)
    __device__ __forceinline__ double *row(int64_t IJ) const { return out + IJ * (IJ + 1) / 2; }
    // bra and ket each of two shells, and no shell the highest of both: every
    // component's canonical order is that of the shells
    __device__ __forceinline__ static bool plain(const QCtx &q)
    {
        return q.sa != q.sb && q.sc != q.sd && max(q.fa, q.fb) != max(q.fc, q.fd);
    }
    // one component of any quartet, if canonical
    __device__ __forceinline__ void one(const QCtx &q, int fi, int fj, int fk, int fl, double v) const
    {
        if ((q.sa == q.sb && fi < fj) || (q.sc == q.sd && fk < fl)) return;
        const int64_t IJ = fpair(fi, fj), KL = fpair(fk, fl);
        if (q.bra == q.ket && IJ < KL) return;
        const double w = v * fscale[fi] * fscale[fj] * fscale[fk] * fscale[fl];
        *(IJ > KL ? row(IJ) + KL : row(KL) + IJ) = w;
    }
    template <int LA, int LB, int LC, int LD, typename R>
    __device__ __forceinline__ void thread_quartet(const QCtx &q, const R *acc, int, bool live) const
    {
        constexpr int NA = ncart(LA), NB = ncart(LB), NC = ncart(LC), ND = ncart(LD), NCD = NC * ND;
        if (!live) return;
        if (!plain(q)) {
#pragma unroll
            for (int t = 0; t < NA * NB * NCD; ++t)
                one(q, q.fa + t / NCD / NB, q.fb + t / NCD % NB, q.fc + t % NCD / ND, q.fd + t % ND, (double)acc[t]);
        } else if (max(q.fa, q.fb) > max(q.fc, q.fd)) {
#pragma unroll
            for (int ab = 0; ab < NA * NB; ++ab) {
                const int fi = q.fa + ab / NB, fj = q.fb + ab % NB;
                double *r = row(fpair(fi, fj));
                const double s = __ldg(fscale + fi) * __ldg(fscale + fj);
                if (q.fc > q.fd) {
#pragma unroll
                    for (int c = 0; c < NC; ++c)
                        run<ND, 1>(r + fpair(q.fc + c, q.fd), acc + ab * NCD + c * ND, q.fd, s * __ldg(fscale + q.fc + c));
                } else {
#pragma unroll
                    for (int d = 0; d < ND; ++d)
                        run<NC, ND>(r + fpair(q.fd + d, q.fc), acc + ab * NCD + d, q.fc, s * __ldg(fscale + q.fd + d));
                }
            }
        } else {
#pragma unroll
            for (int cd = 0; cd < NCD; ++cd)
                ket_row<NA, NB, NCD>(q, q.fc + cd / ND, q.fd + cd % ND, acc + cd);
        }
    }
    // row (fk, fl) of a plain quartet whose ket is the higher pair; x[ab * S]
    template <int NA, int NB, int S, typename R>
    __device__ __forceinline__ void ket_row(const QCtx &q, int fk, int fl, const R *x) const
    {
        double *r = row(fpair(fk, fl));
        const double s = __ldg(fscale + fk) * __ldg(fscale + fl);
        if (q.fa > q.fb) {
#pragma unroll
            for (int a = 0; a < NA; ++a)
                run<NB, S>(r + fpair(q.fa + a, q.fb), x + a * NB * S, q.fb, s * __ldg(fscale + q.fa + a));
        } else {
#pragma unroll
            for (int b = 0; b < NB; ++b)
                run<NA, NB * S>(r + fpair(q.fb + b, q.fa), x + b * S, q.fa, s * __ldg(fscale + q.fb + b));
        }
    }
    template <int LA, int LB, int LC, int LD, int NCW>
    __device__ __forceinline__ void lane_quartet(const QCtx &q, int ic, int id, int, bool live, double *acc, double *) const
    {
        constexpr int NA = ncart(LA), NB = ncart(LB);
        const int fk = q.fc + ic, fl = q.fd + id;
        if (!live) return;
        if (!plain(q)) {
#pragma unroll
            for (int ab = 0; ab < NA * NB; ++ab) one(q, q.fa + ab / NB, q.fb + ab % NB, fk, fl, acc[ab]);
        } else if (max(q.fa, q.fb) > max(q.fc, q.fd)) {
            // neighbouring lanes hold neighbouring elements
            const int64_t KL = fpair(fk, fl);
            const double skl = __ldg(fscale + fk) * __ldg(fscale + fl);
#pragma unroll
            for (int ab = 0; ab < NA * NB; ++ab) {
                const int fi = q.fa + ab / NB, fj = q.fb + ab % NB;
                row(fpair(fi, fj))[KL] = acc[ab] * (skl * __ldg(fscale + fi) * __ldg(fscale + fj));
            }
        } else {
            ket_row<NA, NB, 1>(q, fk, fl, acc);
        }
    }
};

// Runs of equal keys over the lanes of a warp (the thread-mode item lists
// are ordered so that neighbouring lanes often share a bra pair and a ket
// shell): sum() is an inclusive segmented scan, so the last lane of a run
// holds the run's total and issues one atomic for the whole run.  Every lane
// of the warp must take part.
struct WarpRuns {
    unsigned f;   // bit s: lane - 2^s lies in this lane's run
    int steps;    // scan steps that reach the longest run of the warp
    bool last;    // last lane of its run
    __device__ __forceinline__ WarpRuns(int key_hi, int key_lo, int lane)
    {
        // a run is a maximal block of consecutive lanes with one key (the
        // same key may come back later in the warp as another run): the run
        // heads of the warp as one ballot
        const int ph = __shfl_up_sync(0xffffffffu, key_hi, 1), pl = __shfl_up_sync(0xffffffffu, key_lo, 1);
        const bool head = lane == 0 || ph != key_hi || pl != key_lo;
        const unsigned heads = __ballot_sync(0xffffffffu, head);
        const int back = __clz((heads << (31 - lane)));   // lanes since this lane's head
        f = 0;
#pragma unroll
        for (int s = 0; s < 5; ++s)
            if (back >= (1 << s)) f |= 1u << s;
        steps = 32 - __clz((int)__reduce_max_sync(0xffffffffu, (unsigned)back));
        last = lane == 31 || ((heads >> ((lane + 1) & 31)) & 1u);
    }
    template <typename V> __device__ __forceinline__ V sum(V x) const
    {
#pragma unroll
        for (int s = 0; s < 5; ++s) {
            if (s >= steps) break;   // uniform over the warp
            const V y = __shfl_up_sync(0xffffffffu, x, 1 << s);
            if ((f >> s) & 1u) x += y;
        }
        return x;
    }
};

// Full-warp sums of K values per lane (K <= 32) by recursive halving: at each
// of the first log2(KP) butterfly levels (KP = K rounded up to a power of two)
// every lane keeps half of its remaining values and adds its partner's half
// of them, then the remaining levels are a plain butterfly.  Lane L ends with
// the warp's sum of value idx(L) (the kept halves), held by the 32/KP lanes
// that agree on those bits; (KP - 1) + (5 - log2 KP) shuffles in place of the
// 5 K of K separate sums.  Every lane of the warp must take part.
template <int K, typename V>
__device__ __forceinline__ V warp_sum_transposed(const V *v, int lane, int &idx)
{
    constexpr int KP = K <= 1 ? 1 : K <= 2 ? 2 : K <= 4 ? 4 : K <= 8 ? 8 : K <= 16 ? 16 : 32;
    V w[KP];
#pragma unroll
    for (int j = 0; j < KP; ++j) w[j] = j < K ? v[j] : (V)0;
    idx = 0;
    int o = 16;
#pragma unroll
    for (int n = KP; n > 1; n >>= 1, o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (int j = 0; j < n / 2; ++j) {
            const V keep = up ? w[j + n / 2] : w[j], send = up ? w[j] : w[j + n / 2];
            w[j] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
        if (up) idx += n / 2;
    }
#pragma unroll
    for (; o > 0; o >>= 1) w[0] += __shfl_xor_sync(0xffffffffu, w[0], o);
    return w[0];
}

// Direct J/K digestion of unique quartets with 8-fold degeneracy weights:
//   Jacc[i,j] += 2 v' D_kl,  Jacc[k,l] += 2 v' D_ij,
//   Kacc[i,k] += v' D_jl, Kacc[i,l] += v' D_jk, Kacc[j,k] += v' D_il, Kacc[j,l] += v' D_ik,
// v' = v * comp_weight; then J = Jacc + Jacc^T, K = Kacc + Kacc^T reproduce
// J_ij = sum_kl (ij|kl) D_kl and K_ij = sum_kl (ik|jl) D_kl of
// PyQuante/Ints.py:195-223 for symmetric D.
//
// The integrals here are those of the shells' common contraction (no
// per-component scale r_f): D is the pre-scaled density D'_kl = r_k r_l D_kl
// and the caller multiplies J and K by r_i r_j afterwards, which gives the
// same J and K as digesting the scaled integrals with D.
//
// Thread mode: the quartet's six D blocks are loaded once, the six J/K
// blocks (ab, cd, ac, ad, bc, bd) are summed in registers, and each block
// element goes to global memory with one atomic.  Warp mode: see
// lane_quartet.  With NDEN = 2 both
// densities are digested from the same integrals (UHF); WITHK = false keeps
// the Coulomb terms alone.
template <int NDEN, bool WITHK = true>
struct EpiJKn {
    const double *D[NDEN];        // pre-scaled densities
    double *Jacc[NDEN], *Kacc[NDEN];
    const float *Df[NDEN];        // their single-precision copies (FP32 lists of the mixed mode), or null
    ItemScreen scr;               // items skipped by molecule mask or density bound (all fields optional)
    static constexpr bool kCoop = false;   // (its items are cut short by the plan instead)
    __device__ __forceinline__ bool screened(const PairInfo &pb, const PairInfo &pk, int bra, int ket) const
    {
        if (scr.molmask && __ldg(scr.molmask + pb.mol) == 0) return true;
        if (scr.dmax) {
            const double d = fmax(fmax(__ldg(scr.dmax + pb.sa), __ldg(scr.dmax + pb.sb)),
                                  fmax(__ldg(scr.dmax + pk.sa), __ldg(scr.dmax + pk.sb)));
            if (__ldg(scr.Qpair + bra) * __ldg(scr.Qpair + ket) * d < scr.tau) return true;
        }
        return false;
    }
    // this block's copy of the sums
    __device__ __forceinline__ int64_t copy() const { return (int64_t)((int)blockIdx.x & scr.cmask) * scr.cstride; }

    // (called by every lane of the warp; a lane past the end of the item list
    // passes its neighbour's quartet with zero integrals)
    // The per-quartet products, block sums and sums over lanes run in the
    // list's precision R (FP32 lists read the single-precision density); the
    // accumulation into Jacc/Kacc is FP64.
    template <int LA, int LB, int LC, int LD, typename R>
    __device__ __forceinline__ void thread_quartet(const QCtx &q, R *acc, int lane, bool) const
    {
        using T = R;
        constexpr int NA = ncart(LA), NB = ncart(LB), NC = ncart(LC), ND = ncart(LD), NCD = NC * ND;
        // degeneracy weights, applied once; shells of unlike angular momentum, or
        // bra and ket of unlike classes, are never the same, and most warps hold no
        // such quartet at all
        if constexpr (LA == LB || LC == LD || (LA == LC && LB == LD)) {
            const bool bd = LA == LB && q.sa == q.sb, kd = LC == LD && q.sc == q.sd,
                       qd = LA == LC && LB == LD && q.bra == q.ket, af = q.fa > q.fb;
            if (bd || kd || qd) {
#pragma unroll
                for (int a = 0; a < NA; ++a)
#pragma unroll
                    for (int b = 0; b < NB; ++b)
#pragma unroll
                        for (int c = 0; c < NC; ++c)
#pragma unroll
                            for (int d = 0; d < ND; ++d)
                                acc[(a * NB + b) * NCD + c * ND + d] *= (T)comp_weight(a, b, c, d, bd, kd, qd, af);
            }
        }
        // Jacc[a,b] is shared by lanes with the same bra pair; Kacc[a,c] and
        // Kacc[b,c] by lanes that also share the ket's first shell (the bra
        // runs are scanned only for warps of more than one bra pair)
        const WarpRuns rbc(q.bra, q.sc, lane);
        // (the shuffle is taken by every lane, outside any condition)
        const int bra0 = __shfl_sync(0xffffffffu, q.bra, 0);
        const bool one_bra = __all_sync(0xffffffffu, bra0 == q.bra);
        // every density digests the same integrals, one after the other
#pragma unroll
        for (int s = 0; s < NDEN; ++s) {
        const T *Db;
        if constexpr (std::is_same_v<T, float>)
            Db = Df[s] + q.bo;
        else
            Db = D[s] + q.bo;
        double *Jb = Jacc[s] + q.bo + copy(), *Kb = Kacc[s] + q.bo + copy();
        // row bases in 64 bits, offsets within the few rows of a shell in 32
        const int nm = q.nm;
        const int64_t oa = (int64_t)q.fa * nm, ob = (int64_t)q.fb * nm, oc = (int64_t)q.fc * nm;
        const T *Da = Db + oa, *Dbr = Db + ob, *Dc = Db + oc;
        double *Ja = Jb + oa, *Jc = Jb + oc, *Ka = Kb + oa, *Kbr = Kb + ob;
        // Coulomb: Jacc[a,b] and Jacc[c,d]
        {
            T dab[NA][NB], dcd[NC][ND], jcd[NC][ND];
#pragma unroll
            for (int a = 0; a < NA; ++a)
#pragma unroll
                for (int b = 0; b < NB; ++b) dab[a][b] = __ldg(Da + a * nm + q.fb + b);
#pragma unroll
            for (int c = 0; c < NC; ++c)
#pragma unroll
                for (int d = 0; d < ND; ++d) {
                    dcd[c][d] = __ldg(Dc + c * nm + q.fd + d);
                    jcd[c][d] = (T)0;
                }
            T jabv[NA * NB];
#pragma unroll
            for (int a = 0; a < NA; ++a)
#pragma unroll
                for (int b = 0; b < NB; ++b) {
                    T jab = (T)0;
#pragma unroll
                    for (int c = 0; c < NC; ++c)
#pragma unroll
                        for (int d = 0; d < ND; ++d) {
                            const T v = acc[(a * NB + b) * NCD + c * ND + d];
                            jab = fma(v, dcd[c][d], jab);
                            jcd[c][d] = fma(v, dab[a][b], jcd[c][d]);
                        }
                    jabv[a * NB + b] = jab;
                }
            if (NA * NB <= 32 && one_bra) {
                // the whole warp is one bra pair: all NAB sums in one transposed reduction
                int idx;
                const double js = (double)warp_sum_transposed<(NA * NB <= 32 ? NA * NB : 1)>(jabv, lane, idx);
                constexpr int KP = NA * NB <= 1 ? 1 : NA * NB <= 2 ? 2 : NA * NB <= 4 ? 4 : NA * NB <= 8 ? 8 : NA * NB <= 16 ? 16 : 32;
                if (idx < NA * NB && (lane & (32 / KP - 1)) == 0 && js != 0.0)
                    atomicAdd(Ja + idx / NB * nm + q.fb + idx % NB, 2.0 * js);
            } else {
                const WarpRuns rb(q.bra, 0, lane);
#pragma unroll
                for (int ab = 0; ab < NA * NB; ++ab) {
                    const double js = (double)rb.sum(jabv[ab]);
                    if (rb.last && js != 0.0) atomicAdd(Ja + ab / NB * nm + q.fb + ab % NB, 2.0 * js);
                }
            }
#pragma unroll
            for (int c = 0; c < NC; ++c)
#pragma unroll
                for (int d = 0; d < ND; ++d)
                    if (jcd[c][d] != (T)0) atomicAdd(Jc + c * nm + q.fd + d, 2.0 * (double)jcd[c][d]);
        }
        if constexpr (!WITHK) continue;   // Coulomb only
        // exchange rows of the bra's first shell: Kacc[a,c] += v D_bd, Kacc[a,d] += v D_bc
        {
            T dbd[NB][ND], dbc[NB][NC];
#pragma unroll
            for (int b = 0; b < NB; ++b) {
#pragma unroll
                for (int d = 0; d < ND; ++d) dbd[b][d] = __ldg(Dbr + b * nm + q.fd + d);
#pragma unroll
                for (int c = 0; c < NC; ++c) dbc[b][c] = __ldg(Dbr + b * nm + q.fc + c);
            }
#pragma unroll
            for (int a = 0; a < NA; ++a) {
                T kac[NC], kad[ND];
#pragma unroll
                for (int c = 0; c < NC; ++c) kac[c] = (T)0;
#pragma unroll
                for (int d = 0; d < ND; ++d) kad[d] = (T)0;
#pragma unroll
                for (int b = 0; b < NB; ++b)
#pragma unroll
                    for (int c = 0; c < NC; ++c)
#pragma unroll
                        for (int d = 0; d < ND; ++d) {
                            const T v = acc[(a * NB + b) * NCD + c * ND + d];
                            kac[c] = fma(v, dbd[b][d], kac[c]);
                            kad[d] = fma(v, dbc[b][c], kad[d]);
                        }
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    const double ks = (double)rbc.sum(kac[c]);
                    if (rbc.last && ks != 0.0) atomicAdd(Ka + a * nm + q.fc + c, ks);
                }
#pragma unroll
                for (int d = 0; d < ND; ++d)
                    if (kad[d] != (T)0) atomicAdd(Ka + a * nm + q.fd + d, (double)kad[d]);
            }
        }
        // exchange rows of the bra's second shell: Kacc[b,c] += v D_ad, Kacc[b,d] += v D_ac
        {
            T dad[NA][ND], dac[NA][NC];
#pragma unroll
            for (int a = 0; a < NA; ++a) {
#pragma unroll
                for (int d = 0; d < ND; ++d) dad[a][d] = __ldg(Da + a * nm + q.fd + d);
#pragma unroll
                for (int c = 0; c < NC; ++c) dac[a][c] = __ldg(Da + a * nm + q.fc + c);
            }
#pragma unroll
            for (int b = 0; b < NB; ++b) {
                T kbc[NC], kbd[ND];
#pragma unroll
                for (int c = 0; c < NC; ++c) kbc[c] = (T)0;
#pragma unroll
                for (int d = 0; d < ND; ++d) kbd[d] = (T)0;
#pragma unroll
                for (int a = 0; a < NA; ++a)
#pragma unroll
                    for (int c = 0; c < NC; ++c)
#pragma unroll
                        for (int d = 0; d < ND; ++d) {
                            const T v = acc[(a * NB + b) * NCD + c * ND + d];
                            kbc[c] = fma(v, dad[a][d], kbc[c]);
                            kbd[d] = fma(v, dac[a][c], kbd[d]);
                        }
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    const double ks = (double)rbc.sum(kbc[c]);
                    if (rbc.last && ks != 0.0) atomicAdd(Kbr + b * nm + q.fc + c, ks);
                }
#pragma unroll
                for (int d = 0; d < ND; ++d)
                    if (kbd[d] != (T)0) atomicAdd(Kbr + b * nm + q.fd + d, (double)kbd[d]);
            }
        }
        }
    }

    // Warp mode: a lane holds the NAB integrals of one ket component pair
    // (c, d); a slot's lanes are consecutive, d fastest.  Every output's part is
    // summed in the lane first, then over the slot's d or its NCW c lanes by
    // shuffles (Kacc), or over all of them through buf (Jacc[a,b]; NAB x 33
    // doubles of the warp's shared memory).  Lanes without a live quartet carry
    // zeros.
    template <int N> static __device__ __forceinline__ double strided_sum(double x, int stride)
    {
        // the sum over N lanes (N = 1, 3 or 6) at the given stride, valid in the first
        static_assert(N == 1 || N == 3 || N == 6, "cartesian components of s, p, d");
        if constexpr (N == 6) x += __shfl_down_sync(0xffffffffu, x, 3 * stride);
        if constexpr (N > 1) {
            const double y = __shfl_down_sync(0xffffffffu, x, stride), z = __shfl_down_sync(0xffffffffu, x, 2 * stride);
            x += y + z;
        }
        return x;
    }

    template <int LA, int LB, int LC, int LD, int NCW>
    __device__ __forceinline__ void lane_quartet(const QCtx &q, int c, int d, int lane, bool live, double *acc,
                                                 double *buf) const
    {
        constexpr int NA = ncart(LA), NB = ncart(LB), ND = ncart(LD), NAB = NA * NB, W = NCW * ND;
        const bool c_first = c % NCW == 0;
        if constexpr (LA == LB || LC == LD || (LA == LC && LB == LD)) {
            const bool bd = LA == LB && q.sa == q.sb, kd = LC == LD && q.sc == q.sd,
                       qd = LA == LC && LB == LD && q.bra == q.ket, af = q.fa > q.fb;
            if (bd || kd || qd) {
#pragma unroll
                for (int ab = 0; ab < NAB; ++ab) acc[ab] *= comp_weight(ab / NB, ab % NB, c, d, bd, kd, qd, af);
            }
        }
        if (!live) {
#pragma unroll
            for (int ab = 0; ab < NAB; ++ab) acc[ab] = 0.0;
        }
        const int nm = q.nm;
        const int64_t oa = (int64_t)q.fa * nm, ob = (int64_t)q.fb * nm, oc = (int64_t)(q.fc + c) * nm;
#pragma unroll
        for (int s = 0; s < NDEN; ++s) {
            const double *Db = D[s] + q.bo;
            const double *Da = Db + oa, *Dbr = Db + ob;
            double *Jb = Jacc[s] + q.bo + copy();
            // Jacc[c,d] in the lane, Jacc[a,b] over the slot
            {
                const double dcd = __ldg(Db + oc + q.fd + d);
                double jcd = 0.0;
#pragma unroll
                for (int ab = 0; ab < NAB; ++ab) {
                    jcd = fma(acc[ab], __ldg(Da + ab / NB * nm + q.fb + ab % NB), jcd);
                    buf[ab * 33 + lane] = acc[ab] * dcd;
                }
                if (live && jcd != 0.0) atomicAdd(Jb + oc + q.fd + d, 2.0 * jcd);
                __syncwarp();
                // the slot's lanes step through its NAB sums
                if (live) {
                    const int l0 = lane / W * W;
                    for (int ab = lane - l0; ab < NAB; ab += W) {
                        double x = 0.0;
#pragma unroll
                        for (int k = 0; k < W; ++k) x += buf[ab * 33 + l0 + k];
                        if (x != 0.0) atomicAdd(Jb + oa + ab / NB * nm + q.fb + ab % NB, 2.0 * x);
                    }
                }
                __syncwarp();
            }
            if constexpr (!WITHK) continue;   // Coulomb only
            double *Ka = Kacc[s] + q.bo + copy() + oa, *Kbr = Kacc[s] + q.bo + copy() + ob;
            {
                double dbd[NB], dbc[NB];
#pragma unroll
                for (int b = 0; b < NB; ++b) {
                    dbd[b] = __ldg(Dbr + b * nm + q.fd + d);
                    dbc[b] = __ldg(Dbr + b * nm + q.fc + c);
                }
#pragma unroll
                for (int a = 0; a < NA; ++a) {
                    double kac = 0.0, kad = 0.0;
#pragma unroll
                    for (int b = 0; b < NB; ++b) {
                        kac = fma(acc[a * NB + b], dbd[b], kac);
                        kad = fma(acc[a * NB + b], dbc[b], kad);
                    }
                    kac = strided_sum<ND>(kac, 1);
                    kad = strided_sum<NCW>(kad, ND);
                    if (live && d == 0 && kac != 0.0) atomicAdd(Ka + a * nm + q.fc + c, kac);
                    if (live && c_first && kad != 0.0) atomicAdd(Ka + a * nm + q.fd + d, kad);
                }
            }
            {
                double dad[NA], dac[NA];
#pragma unroll
                for (int a = 0; a < NA; ++a) {
                    dad[a] = __ldg(Da + a * nm + q.fd + d);
                    dac[a] = __ldg(Da + a * nm + q.fc + c);
                }
#pragma unroll
                for (int b = 0; b < NB; ++b) {
                    double kbc = 0.0, kbd = 0.0;
#pragma unroll
                    for (int a = 0; a < NA; ++a) {
                        kbc = fma(acc[a * NB + b], dad[a], kbc);
                        kbd = fma(acc[a * NB + b], dac[a], kbd);
                    }
                    kbc = strided_sum<ND>(kbc, 1);
                    kbd = strided_sum<NCW>(kbd, ND);
                    if (live && d == 0 && kbc != 0.0) atomicAdd(Kbr + b * nm + q.fc + c, kbc);
                    if (live && c_first && kbd != 0.0) atomicAdd(Kbr + b * nm + q.fd + d, kbd);
                }
            }
        }
    }
};

// One density (RHF, or one spin at a time) and two (UHF's alpha and beta
// densities digesting the same integrals in one pass).
using EpiJK = EpiJKn<1>;
using EpiJK2 = EpiJKn<2>;
// Coulomb only (DFT's getJ): no exchange products, no K atomics
using EpiJ = EpiJKn<1, false>;



// Schwarz: Q2[pair] = max over components of |(ij|ij)| (diagonal quartets).
struct EpiSchwarz {
    unsigned long long *Q2bits;   // bit patterns of non-negative doubles
    const double *fscale;
    static constexpr bool kCoop = true;
    __device__ __forceinline__ bool screened(const PairInfo &, const PairInfo &, int, int) const { return false; }
    template <int LC, int LD, typename R>
    __device__ __forceinline__ void ab(const QCtx &q, int ia, int ib, const R *acc) const
    {
        constexpr int ND = ncart(LD), NCD = ncart(LC) * ncart(LD);
        const int cd = ia * ND + ib;   // (ic, id) == (ia, ib) on a diagonal quartet
        double v = 0.0;
#pragma unroll
        for (int c = 0; c < NCD; ++c)
            if (c == cd) v = (double)acc[c];
        const double s = fscale[q.fa + ia] * fscale[q.fb + ib];
        v = fabs(v) * s * s;
        atomicMax(Q2bits + q.bra, (unsigned long long)__double_as_longlong(v));
    }
    template <int LA, int LB, int LC, int LD, typename R>
    __device__ __forceinline__ void thread_quartet(const QCtx &q, const R *acc, int lane, bool live) const
    {
        constexpr int NB = ncart(LB), NCD = ncart(LC) * ncart(LD);
        (void)lane;
        if (!live) return;
#pragma unroll
        for (int ab = 0; ab < ncart(LA) * NB; ++ab) this->ab<LC, LD, R>(q, ab / NB, ab % NB, acc + ab * NCD);
    }
    template <int LA, int LB, int LC, int LD, int NCW>
    __device__ __forceinline__ void lane_quartet(const QCtx &q, int ic, int id, int, bool live, double *acc, double *) const
    {
        // (ia, ib) == (ic, id) on a diagonal quartet
        constexpr int ND = ncart(LD);
        if (!live) return;
        double v = 0.0;
#pragma unroll
        for (int ab = 0; ab < ncart(LA) * ncart(LB); ++ab)
            if (ab == ic * ND + id) v = acc[ab];
        const double s = fscale[q.fc + ic] * fscale[q.fd + id];
        v = fabs(v) * s * s;
        atomicMax(Q2bits + q.bra, (unsigned long long)__double_as_longlong(v));
    }
};

// ------------------------------------------------- Obara--Saika classes --
// Per-primitive-quartet coefficients of the Obara--Saika vertical recurrence
// (PA = P - A, QC = Q - C, WP = -rho/zeta PQ, WQ = rho/eta PQ, PQ = P - Q,
// rz = rho/zeta = eta/(zeta+eta), re = rho/eta = zeta/(zeta+eta),
// oo2z = 1/(2 zeta), oo2e = 1/(2 eta), oo2ze = 1/(2 (zeta+eta))).
template <typename R>
struct OsGeom {
    R PA[3], WP[3], QC[3], WQ[3];
    R oo2z, rz, oo2e, re, oo2ze;
};

// Classes without generated routines keep the Rys quadrature.
template <int LA, int LB, int LC, int LD>
struct OsClass {
    static constexpr bool kOn = false;
    static constexpr int NV = 1;
    template <typename R>
    __device__ static void vrr(const OsGeom<R> &, const R *, R *) {}
    template <typename R>
    __device__ static void hrr(const R *, const R *, const R *, R *) {}
};

#include "os_classes.inc"

// ---------------------------------------------------------- thread mode --
// Register cap per class (via the minimum resident blocks of 128 threads):
// small classes are latency bound, so they trade registers for occupancy
// (six blocks for up to three components, five for up to nine, three for
// the 27 of (11|10), measured faster than fewer even with a few spilled
// registers).
__host__ __device__ constexpr int thread_min_blocks(int nabcd)
{
    return nabcd == 1 ? 8 : (nabcd <= 3 ? 6 : (nabcd <= 9 ? 5 : (nabcd == 27 ? 3 : 2)));
}

struct QuartetGeomF {
    float A[3], C[3], AB[3], CD[3];
};

// FP32 lists of the mixed mode: geometry, F_m(T) and the vertical
// recurrence in single precision, accumulated into the contracted [e0|f0].
template <int LA, int LB, int LC, int LD>
__device__ __forceinline__ void os_prim_quartet_f32(const QuartetGeomF &g, const float *P, const float *Q, float *v)
{
    constexpr int LT = LA + LB + LC + LD;
    const float zeta = P[0], eta = Q[0];
    const float PQ[3] = {P[2] - Q[2], P[3] - Q[3], P[4] - Q[4]};
    const float rs = rsqrtf(zeta + eta), izpe = rs * rs;
    const float T = zeta * eta * izpe * (PQ[0] * PQ[0] + PQ[1] * PQ[1] + PQ[2] * PQ[2]);
    const float pre = P[5] * Q[5] * rs;
    float F[LT + 1];
    boys_os_f32<LT>(T, F);
#pragma unroll
    for (int m = 0; m <= LT; ++m) F[m] *= pre;
    OsGeom<float> o;
    const float rz = eta * izpe, re = zeta * izpe;
#pragma unroll
    for (int x = 0; x < 3; ++x) {
        o.PA[x] = P[2 + x] - g.A[x];
        o.QC[x] = Q[2 + x] - g.C[x];
        o.WP[x] = -rz * PQ[x];
        o.WQ[x] = re * PQ[x];
    }
    o.rz = rz;
    o.re = re;
    o.oo2z = 0.5f * P[1];
    o.oo2e = 0.5f * Q[1];
    o.oo2ze = 0.5f * izpe;
    OsClass<LA, LB, LC, LD>::template vrr<float>(o, F, v);
}

// G lanes share an item (1, or kCoopLanes for the long items of whole
// quartets), each every G-th primitive quartet; the contracted [e0|f0] are
// added over them, and the first lane has the item's epilogue.
template <int LA, int LB, int LC, int LD, typename R, class Epi, int G = 1>
__global__ void __launch_bounds__(128, thread_min_blocks(ncart(LA) * ncart(LB) * ncart(LC) * ncart(LD)))
eri_thread_kernel(const int4 *__restrict__ list, int nq,
                                                         const PairInfo *__restrict__ pairs,
                                                         const PrimPair *__restrict__ prims, Epi epi)
{
    constexpr int NA = ncart(LA), NB = ncart(LB), NC = ncart(LC), ND = ncart(LD);
    constexpr int NAB = NA * NB, NCD = NC * ND;
    using OS = OsClass<LA, LB, LC, LD>;
    static_assert(OS::kOn, "thread mode has the Obara--Saika classes only");
    // whole warps step through the list together (the J/K epilogue reduces
    // over the lanes); a lane past the end repeats the last item with no
    // primitive quartets
    const int lane = threadIdx.x & 31;
    for (int base = (blockIdx.x * blockDim.x + threadIdx.x - lane) / G; base < nq; base += gridDim.x * blockDim.x / G) {
        const int qi = base + lane / G;
        const bool live = qi < nq;
        int4 e = list[live ? qi : nq - 1];   // bra pair, ket pair, first primitive quartet, count
        if (!live) e.w = 0;
        const PairInfo &pb = pairs[e.x];
        const PairInfo &pk = pairs[e.y];
        // screened items (masked molecules, small density bounds) carry no
        // primitive quartets; a warp with none left skips the item altogether
        const bool skip = live && epi.screened(pb, pk, e.x, e.y);
        if (__all_sync(0xffffffffu, skip || !live)) continue;
        if (skip) e.w = 0;
        const double Ax = pb.A[0], Ay = pb.A[1], Az = pb.A[2];
        const double Cx = pk.A[0], Cy = pk.A[1], Cz = pk.A[2];
        const double ABx = pb.AB[0], ABy = pb.AB[1], ABz = pb.AB[2];
        const double CDx = pk.AB[0], CDy = pk.AB[1], CDz = pk.AB[2];
        R acc[NAB * NCD];
#pragma unroll
        for (int c = 0; c < NAB * NCD; ++c) acc[c] = (R)0;
        // primitive quartet g of the item = (bra primitive g % npb, ket
        // primitive g / npb): the bra index runs fastest, so the lanes of a
        // warp (which share the bra pair) step through the same bra
        // primitives and each lane fetches its own ket primitive pair only
        // once per npb steps
        const int npb = pb.nprim;
        const PrimPair *pbp = prims + pb.prim_off, *pkp = prims + pk.prim_off;
        int ik = e.z / npb, ib = e.z - (e.z / npb) * npb;
        if constexpr (std::is_same_v<R, float>) {
            // FP32 list of the mixed mode: single-precision primitive data
            QuartetGeomF gf;
#pragma unroll
            for (int x = 0; x < 3; ++x) {
                gf.A[x] = (float)pb.A[x];
                gf.C[x] = (float)pk.A[x];
                gf.AB[x] = (float)pb.AB[x];
                gf.CD[x] = (float)pk.AB[x];
            }
            float Pn[8], Q[8];
            ld8f(pbp[ib].f, Pn);
            ld8f(pkp[ik].f, Q);
            float v[OS::NV];
#pragma unroll
            for (int c = 0; c < OS::NV; ++c) v[c] = 0.0f;
            for (int t = 0; t < e.w; ++t) {
                float P[8];
#pragma unroll
                for (int c = 0; c < 8; ++c) P[c] = Pn[c];
                int ib2 = ib + 1, ik2 = ik;
                if (ib2 == npb) {
                    ib2 = 0;
                    ++ik2;
                }
                if (t + 1 < e.w) ld8f(pbp[ib2].f, Pn);
                float Qn[8];
                if (ik2 != ik && t + 1 < e.w) ld8f(pkp[ik2].f, Qn);
                os_prim_quartet_f32<LA, LB, LC, LD>(gf, P, Q, v);
                if (ik2 != ik && t + 1 < e.w) {
#pragma unroll
                    for (int c = 0; c < 8; ++c) Q[c] = Qn[c];
                }
                ib = ib2;
                ik = ik2;
            }
            OS::template hrr<float>(gf.AB, gf.CD, v, reinterpret_cast<float *>(acc));
            const QCtx q = make_qctx(pb, pk, e.x, e.y);
            epi.template thread_quartet<LA, LB, LC, LD, R>(q, acc, lane, live);
            continue;
        }
        // Obara--Saika per primitive quartet, Head-Gordon--Pople transfer
        // once per item on the contracted [e0|f0]
        constexpr int LT = LA + LB + LC + LD;
        R v[OS::NV];
#pragma unroll
        for (int c = 0; c < OS::NV; ++c) v[c] = (R)0;
        const auto add = [&](const PrimJK &P, const PrimJK &Q) {
            const double zeta = P.zeta, eta = Q.zeta;
            const double PQx = P.P[0] - Q.P[0], PQy = P.P[1] - Q.P[1], PQz = P.P[2] - Q.P[2];
            const double rs = rsqrt_nr_unchecked(zeta + eta);   // exponent sums: 1e-36 < x < 1e36
            const double izpe = rs * rs;
            const double T = zeta * eta * izpe * (PQx * PQx + PQy * PQy + PQz * PQz);
            const double pre = P.K * Q.K * rs;
            double F[LT + 1];
            boys_os<LT>(T, F);
            R Fs[LT + 1];
#pragma unroll
            for (int m = 0; m <= LT; ++m) Fs[m] = (R)(F[m] * pre);
            OsGeom<R> g;
            const double rz = eta * izpe, re = zeta * izpe;
            g.PA[0] = P.P[0] - Ax;
            g.PA[1] = P.P[1] - Ay;
            g.PA[2] = P.P[2] - Az;
            g.QC[0] = Q.P[0] - Cx;
            g.QC[1] = Q.P[1] - Cy;
            g.QC[2] = Q.P[2] - Cz;
            g.WP[0] = -rz * PQx;
            g.WP[1] = -rz * PQy;
            g.WP[2] = -rz * PQz;
            g.WQ[0] = re * PQx;
            g.WQ[1] = re * PQy;
            g.WQ[2] = re * PQz;
            g.rz = rz;
            g.re = re;
            g.oo2z = 0.5 * P.izeta;
            g.oo2e = 0.5 * Q.izeta;
            g.oo2ze = 0.5 * izpe;
            OS::template vrr<R>(g, Fs, v);
        };
        if constexpr (G > 1) {
            for (int t = lane % G; t < e.w; t += G) {
                const int kq = (e.z + t) / npb, kb = e.z + t - kq * npb;
                add(load_prim_jk(pbp + kb), load_prim_jk(pkp + kq));
            }
            __syncwarp();
#pragma unroll
            for (int c = 0; c < OS::NV; ++c)
#pragma unroll
                for (int o = G / 2; o > 0; o >>= 1) v[c] += __shfl_xor_sync(0xffffffffu, v[c], o);
        } else {
            PrimJK Pn = load_prim_jk(pbp + ib);
            PrimJK Q = load_prim_jk(pkp + ik);
            for (int t = 0; t < e.w; ++t) {
                const PrimJK P = Pn;
                int ib2 = ib + 1, ik2 = ik;
                if (ib2 == npb) {
                    ib2 = 0;
                    ++ik2;
                }
                if (t + 1 < e.w) Pn = load_prim_jk(pbp + ib2);
                // the next ket primitive pair, fetched a step ahead
                PrimJK Qn = Q;
                if (ik2 != ik && t + 1 < e.w) Qn = load_prim_jk(pkp + ik2);
                add(P, Q);
                Q = Qn;
                ib = ib2;
                ik = ik2;
            }
        }
        const R AB[3] = {(R)ABx, (R)ABy, (R)ABz}, CD[3] = {(R)CDx, (R)CDy, (R)CDz};
        OS::template hrr<R>(AB, CD, v, acc);
        const QCtx q = make_qctx(pb, pk, e.x, e.y);
        epi.template thread_quartet<LA, LB, LC, LD, R>(q, acc, lane, live && lane % G == 0);
    }
}

// ------------------------------------------------------------ warp mode --
// The larger classes, by Rys quadrature.  A warp holds S = 32/NCD quartets
// (two halves of (22|22)'s ket components take turns); a pass takes up to PB
// primitive quartets of each through three steps with a warp barrier between
// them: roots and recurrence coefficients (a lane per primitive quartet,
// quartet and root), 2-D integrals into shared memory (times three axes), and
// assembly, where a lane adds up the NAB bra components of its ket component
// pair in registers (its 2-D entries are at compile-time offsets from one
// address per axis).
// Bound by shared-memory wavefronts (70-77 % of the L1 data pipe before the
// pitches were odd) and FP64 issue (28 % of its peak; 10-19 % before).  C8H18 /
// 6-31G** (N = 210), the eight classes one after the other, launches included:
// 794 us, of which (21|11) 185; with 256-thread blocks whose eight warps met at
// two block barriers a pass, and a digestion through a shared tile, 1077 and 329.
// The whole build: 2.38 -> 2.13 ms; (H2O)8 / 6-31G** 0.372 -> 0.324 ms.  16 KB of
// tables a warp (longer passes, fewer blocks) measured the same.
constexpr int kWarpsPerBlock = 4;

template <int LA, int LB, int LC, int LD>
struct WarpLayout {
    static constexpr int NAB = ncart(LA) * ncart(LB), NC = ncart(LC), ND = ncart(LD), NCD = NC * ND;
    static constexpr int NR = (LA + LB + LC + LD) / 2 + 1;
    static constexpr int HALVES = NCD > 32 ? 2 : 1, NCW = NC / HALVES, W = NCW * ND, S = 32 / W;
    // odd pitches: the lanes' tables (2-D step) and the slots' (assembly) spread over the banks
    static constexpr int G2D = ((LA + 1) * (LB + 1) * (LC + 1) * (LD + 1)) | 1, slot_words = 3 * NR * G2D | 1;
    // primitive quartets of a pass: their roots occupy the lanes, within 12 KB of tables
    static constexpr int fit = 32 / (S * NR), by_mem = 12288 / (8 * S * slot_words);
    static constexpr int PB0 = fit < by_mem ? fit : by_mem, PB = PB0 < 1 ? 1 : (PB0 > 4 ? 4 : PB0);
    static constexpr int tab_words = PB * S * slot_words;
    // the Jacc[a,b] sums reuse the tables
    static constexpr int words = tab_words > NAB * 33 ? tab_words : NAB * 33;
    static constexpr size_t bytes = sizeof(double) * kWarpsPerBlock * words;
};

template <int NR> struct RysRoots {
    double w[NR], b00[NR], b10[NR], b01[NR], ce[NR], cz[NR];
    double PA[3], QC[3], PQ[3];
};
struct SlotData {
    QCtx q;
    int npb, pp0, npp, pb_off, pk_off;
    bool live;         // a work item that is not screened
    double A[3], AB[3], C[3], CD[3];
};

template <int LA, int LB, int LC, int LD, class Epi>
__global__ void __launch_bounds__(kWarpsPerBlock * 32, WarpLayout<LA, LB, LC, LD>::NAB > 18 ? 3 : 4) eri_warp_kernel(const int4 *__restrict__ list, int nq,
                                                                          const PairInfo *__restrict__ pairs,
                                                                          const PrimPair *__restrict__ prims, Epi epi)
{
    using Lay = WarpLayout<LA, LB, LC, LD>;
    constexpr int NB = ncart(LB), ND = Lay::ND, NAB = Lay::NAB, NR = Lay::NR, G2D = Lay::G2D, S = Lay::S, W = Lay::W,
                  PB = Lay::PB, SW = Lay::slot_words;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ SlotData sd[kWarpsPerBlock][S];
    __shared__ RysRoots<NR> sr[kWarpsPerBlock][PB * S];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double *tab = reinterpret_cast<double *>(smem_raw) + (size_t)warp * Lay::words;
    const int slot = lane / W, k = lane - slot * W;
    const int stride = gridDim.x * kWarpsPerBlock * S;
    for (int base = (blockIdx.x * kWarpsPerBlock + warp) * S; base < nq; base += stride) {
        int npp = 0;
        bool any = false;
        if (lane < S) {
            // (a slot without a live item keeps a valid quartet and no primitives)
            const int qi = base + lane;
            const int4 e = list[qi < nq ? qi : nq - 1];
            const PairInfo &pb = pairs[e.x];
            const PairInfo &pk = pairs[e.y];
            SlotData &s = sd[warp][lane];
            s.live = qi < nq && !epi.screened(pb, pk, e.x, e.y);
            any = s.live;
            npp = s.live ? e.w : 0;   // (0 too where every primitive pair was dropped: zero integrals)
            s.q = make_qctx(pb, pk, e.x, e.y);
            s.npb = pb.nprim;
            s.pp0 = e.z;
            s.npp = npp;
            s.pb_off = pb.prim_off;
            s.pk_off = pk.prim_off;
#pragma unroll
            for (int x = 0; x < 3; ++x) {
                s.A[x] = pb.A[x];
                s.AB[x] = pb.AB[x];
                s.C[x] = pk.A[x];
                s.CD[x] = pk.AB[x];
            }
        }
        const int maxpp = (int)__reduce_max_sync(0xffffffffu, (unsigned)npp);
        if (!__any_sync(0xffffffffu, any)) continue;   // nothing but screened items
        __syncwarp();
        const bool live = slot < S && sd[warp][slot < S ? slot : 0].live;
#pragma unroll 1
        for (int half = 0; half < Lay::HALVES; ++half) {
            const int c = half * Lay::NCW + k / ND, d = k - k / ND * ND;
            const int ox = cart_l(LC, c, 0) * (LD + 1) + cart_l(LD, d, 0);
            const int oy = cart_l(LC, c, 1) * (LD + 1) + cart_l(LD, d, 1);
            const int oz = cart_l(LC, c, 2) * (LD + 1) + cart_l(LD, d, 2);
            double acc[NAB];
#pragma unroll
            for (int ab = 0; ab < NAB; ++ab) acc[ab] = 0.0;
            for (int pp0 = 0; pp0 < maxpp; pp0 += PB) {
                const int nb = maxpp - pp0 < PB ? maxpp - pp0 : PB;
                if (lane < nb * S * NR) {
                    const int bs = lane / NR, r = lane - bs * NR, b = bs / S;
                    const SlotData &s = sd[warp][bs - b * S];
                    if (pp0 + b < s.npp) {
                        // bra primitives fastest
                        const int g = s.pp0 + pp0 + b, jk = g / s.npb, jb = g - jk * s.npb;
                        const PrimJK P = load_prim_jk(prims + s.pb_off + jb), Q = load_prim_jk(prims + s.pk_off + jk);
                        const double PQ[3] = {P.P[0] - Q.P[0], P.P[1] - Q.P[1], P.P[2] - Q.P[2]};
                        const double rs = rsqrt_nr(P.zeta + Q.zeta), izpe = rs * rs;
                        const double T = P.zeta * Q.zeta * izpe * (PQ[0] * PQ[0] + PQ[1] * PQ[1] + PQ[2] * PQ[2]);
                        double u, w;
                        rys_root(NR, r, T, u, w);
                        const RysCoef f = rys_coef(u, P.zeta, Q.zeta, P.izeta, Q.izeta, izpe);
                        RysRoots<NR> &o = sr[warp][bs];
                        o.w[r] = w * P.K * Q.K * rs;
                        o.b00[r] = f.b00;
                        o.b10[r] = f.b10;
                        o.b01[r] = f.b01;
                        o.ce[r] = f.ce;
                        o.cz[r] = f.cz;
                        if (r == 0) {
#pragma unroll
                            for (int x = 0; x < 3; ++x) {
                                o.PA[x] = P.P[x] - s.A[x];
                                o.QC[x] = Q.P[x] - s.C[x];
                                o.PQ[x] = PQ[x];
                            }
                        }
                    }
                }
                __syncwarp();
                for (int t = lane; t < nb * S * NR * 3; t += 32) {
                    const int bs = t / (NR * 3), rx = t - bs * (NR * 3), r = rx / 3, x = rx - r * 3, b = bs / S;
                    const SlotData &s = sd[warp][bs - b * S];
                    if (pp0 + b < s.npp) {
                        const RysRoots<NR> &o = sr[warp][bs];
                        const RysCoef f{o.b00[r], o.b10[r], o.b01[r], o.ce[r], o.cz[r]};
                        rys2d_c<LA, LB, LC, LD, double>(f, o.PA[x], o.QC[x], o.PQ[x], s.AB[x], s.CD[x],
                                                        x == 0 ? o.w[r] : 1.0, tab + bs * SW + (x * NR + r) * G2D);
                    }
                }
                __syncwarp();
                if (live) {
                    const int left = sd[warp][slot].npp - pp0, mine = left < nb ? left : nb;
#pragma unroll 1
                    for (int b = 0; b < mine; ++b) {
                        const double *gx = tab + (b * S + slot) * SW + ox, *gy = tab + (b * S + slot) * SW + NR * G2D + oy,
                                     *gz = tab + (b * S + slot) * SW + 2 * NR * G2D + oz;
#pragma unroll 1
                        for (int r = 0; r < NR; ++r, gx += G2D, gy += G2D, gz += G2D) {
                            // entries (a, b') of each axis: one address, compile-time offsets
                            double X[(LA + 1) * (LB + 1)], Y[(LA + 1) * (LB + 1)], Z[(LA + 1) * (LB + 1)];
#pragma unroll
                            for (int m = 0; m < (LA + 1) * (LB + 1); ++m) {
                                X[m] = gx[m * (LC + 1) * (LD + 1)];
                                Y[m] = gy[m * (LC + 1) * (LD + 1)];
                                Z[m] = gz[m * (LC + 1) * (LD + 1)];
                            }
#pragma unroll
                            for (int ab = 0; ab < NAB; ++ab) {
                                const int ia = ab / NB, ib = ab % NB;
                                acc[ab] = fma(X[cart_lx(LA, ia) * (LB + 1) + cart_lx(LB, ib)] *
                                                  Y[cart_ly(LA, ia) * (LB + 1) + cart_ly(LB, ib)],
                                              Z[cart_lz(LA, ia) * (LB + 1) + cart_lz(LB, ib)], acc[ab]);
                            }
                        }
                    }
                }
                __syncwarp();   // the next pass, or the epilogue's buffer, overwrites the tables
            }
            epi.template lane_quartet<LA, LB, LC, LD, Lay::NCW>(sd[warp][slot < S ? slot : 0].q, c, d, lane, live, acc,
                                                                tab);
        }
        __syncwarp();   // the next items overwrite the slots
    }
}

// ------------------------------------------------------------- dispatch --
template <int LA, int LB, int LC, int LD>
struct ClassTag {};

__host__ __device__ constexpr int pc_la(int c) { return c == 0 ? 0 : (c <= 2 ? 1 : 2); }
__host__ __device__ constexpr int pc_lb(int c) { return c == 0 ? 0 : (c == 1 ? 0 : (c == 2 ? 1 : c - 3)); }

template <int LA, int LB, int LC, int LD, typename R, class Epi>
inline cudaError_t launch_eri_class(const int4 *list, int nq, const PairInfo *pairs, const PrimPair *prims,
                                    const Epi &epi, cudaStream_t st, int nsm, int nlong)
{
    if (nq <= 0) return cudaSuccess;
    constexpr int NAB = ncart(LA) * ncart(LB), NCD = ncart(LC) * ncart(LD);
    if constexpr (NAB * NCD <= kThreadMax) {
        if constexpr (Epi::kCoop) {
            // the list's first nlong items, of more than kCoopItem primitive quartets
            if (nlong > 0) {
                const int grid = grid_blocks(nlong, 128 / kCoopLanes, nsm * 32);
                eri_thread_kernel<LA, LB, LC, LD, R, Epi, kCoopLanes><<<grid, 128, 0, st>>>(list, nlong, pairs, prims,
                                                                                            epi);
                list += nlong;
                nq -= nlong;
            }
            if (nq == 0) return cudaGetLastError();
        }
        const int grid = grid_blocks(nq, 128, nsm * 32);
        eri_thread_kernel<LA, LB, LC, LD, R, Epi><<<grid, 128, 0, st>>>(list, nq, pairs, prims, epi);
    } else if constexpr (std::is_same_v<R, double>) {
        using Lay = WarpLayout<LA, LB, LC, LD>;
        auto kern = eri_warp_kernel<LA, LB, LC, LD, Epi>;
        // the attribute is per device: set once per instantiation and device
        static std::atomic<unsigned long long> attr_set{0};
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return e;
        const unsigned long long bit = dev < 64 ? 1ull << dev : 0ull;
        if (!bit || !(attr_set.load() & bit)) {
            e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Lay::bytes);
            if (e != cudaSuccess) return e;
            attr_set.fetch_or(bit);
        }
        const int grid = grid_blocks(nq, kWarpsPerBlock * Lay::S, nsm * 16);
        kern<<<grid, kWarpsPerBlock * 32, Lay::bytes, st>>>(list, nq, pairs, prims, epi);
    } else {
        return cudaErrorInvalidValue;   // the host sends these classes' FP32 lists to the FP64 kernels
    }
    return cudaGetLastError();
}

// Run class `qc` (0..20): bra pair class cb >= ket pair class ck.
template <typename R, class Epi>
inline cudaError_t launch_eri(int qc, const int4 *list, int nq, const PairInfo *pairs, const PrimPair *prims,
                              const Epi &epi, cudaStream_t st, int nsm, int nlong = 0)
{
#define PQB_CASE(CB, CK)                                                                                       \
    case CB *(CB + 1) / 2 + CK:                                                                               \
        return launch_eri_class<pc_la(CB), pc_lb(CB), pc_la(CK), pc_lb(CK), R, Epi>(list, nq, pairs, prims, epi, \
                                                                                    st, nsm, nlong);
    switch (qc) {
        PQB_CASE(0, 0)
        PQB_CASE(1, 0) PQB_CASE(1, 1)
        PQB_CASE(2, 0) PQB_CASE(2, 1) PQB_CASE(2, 2)
        PQB_CASE(3, 0) PQB_CASE(3, 1) PQB_CASE(3, 2) PQB_CASE(3, 3)
        PQB_CASE(4, 0) PQB_CASE(4, 1) PQB_CASE(4, 2) PQB_CASE(4, 3) PQB_CASE(4, 4)
        PQB_CASE(5, 0) PQB_CASE(5, 1) PQB_CASE(5, 2) PQB_CASE(5, 3) PQB_CASE(5, 4) PQB_CASE(5, 5)
    }
#undef PQB_CASE
    return cudaErrorInvalidValue;
}

}  // namespace pqb
