// Work items are int4 {bra pair, ket pair, first primitive quartet, count}:
// a shell quartet's primitive quartets (bra-major, ket-minor) may be split
// over several items whose contributions add (J/K digestion is linear).
// Host-side entry points into the class-templated ERI engine (the direct J/K
// ones take the pre-scaled density D'_kl = r_k r_l D_kl, see EpiJK, and an
// optional item screen, see ItemScreen), one per
// (epilogue, precision) combination; each lives in its own translation unit
// so the 21 class instantiations compile in parallel.
#pragma once
#include <cuda_runtime.h>

#include "pqb_types.h"

namespace pqb {
struct EpiPacked;
template <int NDEN, bool WITHK> struct EpiJKn;
struct EpiSchwarz;

// nlong: the list's leading items of more than kCoopItem primitive quartets
cudaError_t launch_packed_f64(int qc, const int4 *list, int nq, int nlong, const PairInfo *pairs,
                              const PrimPair *prims, double *out, const double *fscale, cudaStream_t st, int nsm);
cudaError_t launch_jk_f64(int qc, const int4 *list, int nq, const PairInfo *pairs, const PrimPair *prims,
                          const double *Dscaled, double *Jacc, double *Kacc, int n, cudaStream_t st, int nsm,
                          const ItemScreen &scr = ItemScreen{});
cudaError_t launch_jk_f32(int qc, const int4 *list, int nq, const PairInfo *pairs, const PrimPair *prims,
                          const double *Dscaled, const float *Dscaled_f, double *Jacc, double *Kacc, int n,
                          cudaStream_t st, int nsm, const ItemScreen &scr = ItemScreen{});
// J alone (the Coulomb digestion, no exchange)
cudaError_t launch_j_f64(int qc, const int4 *list, int nq, const PairInfo *pairs, const PrimPair *prims,
                         const double *Dscaled, double *Jacc, cudaStream_t st, int nsm, const ItemScreen &scr = ItemScreen{});
cudaError_t launch_j_f32(int qc, const int4 *list, int nq, const PairInfo *pairs, const PrimPair *prims,
                         const double *Dscaled, const float *Dscaled_f, double *Jacc, cudaStream_t st, int nsm,
                         const ItemScreen &scr = ItemScreen{});
// two densities (UHF alpha and beta) digesting the same integrals
cudaError_t launch_jk2_f64(int qc, const int4 *list, int nq, const PairInfo *pairs, const PrimPair *prims,
                           const double *const Dscaled[2], double *const Jacc[2], double *const Kacc[2],
                           cudaStream_t st, int nsm, const ItemScreen &scr = ItemScreen{});
cudaError_t launch_jk2_f32(int qc, const int4 *list, int nq, const PairInfo *pairs, const PrimPair *prims,
                           const double *const Dscaled[2], const float *const Dscaled_f[2], double *const Jacc[2],
                           double *const Kacc[2], cudaStream_t st, int nsm, const ItemScreen &scr = ItemScreen{});
cudaError_t launch_schwarz_f64(int qc, const int4 *list, int nq, int nlong, const PairInfo *pairs,
                               const PrimPair *prims, unsigned long long *Q2bits, const double *fscale, cudaStream_t st, int nsm);
// Coulomb matrix alone in the Hermite basis (eri_jengine.cu): the primitive
// pairs of each L = La + Lb (n[L] from off[L] of list, sorted by the shell
// pair's Schwarz factor, descending), and their Hermite density H and potential
// V (nherm(L) values each from hoff[L]).
struct JPrim {
    double zeta, P[3], Q;
    int pair, prim;
};
struct JLists {
    JPrim *list = nullptr;
    double *H = nullptr, *V = nullptr;
    int n[5] = {0}, off[5] = {0};
    int64_t hoff[5] = {0}, words = 0;
};
cudaError_t launch_hermite_pairs(int n, const int2 *src, const PairInfo *pairs, const PrimPair *prims, const double *Q,
                                 JPrim *out, cudaStream_t st);
cudaError_t launch_hermite_density(int L, const JLists &l, const PairInfo *pairs, const PrimPair *prims, const double *D,
                                   int nbf, cudaStream_t st);
cudaError_t launch_hermite_coulomb(int LP, int LQ, const JLists &l, double thresh, cudaStream_t st, int nsm);
// first[pair]: offset of the pair's V
cudaError_t launch_hermite_fock(int npair, const PairInfo *pairs, const PrimPair *prims, const int64_t *first,
                                const double *V, int nbf, const double *escale, double *J, cudaStream_t st);
// Adds dE2 per shell (gshell[kGradCopies][3 nshell], a block its copy) from the
// pre-scaled density; the gather adds the copies and the shells to their atoms.
constexpr int kGradCopies = 64;
cudaError_t launch_grad(int qc, const int4 *list, int nq, const PairInfo *pairs, const PrimPair *prims,
                        const double *Dscaled, double *gshell, int nshell, cudaStream_t st, int nsm);
cudaError_t launch_grad_gather(int nshell, const int *shell_atom, const double *gshell, double *grad, cudaStream_t st);
}  // namespace pqb
