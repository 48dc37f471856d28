// Device-resident data layout of a basis (built by the host in pqb_capi.cu).
//
// Shell pairs are stored once per unordered pair of shells, oriented so the
// first shell has the higher angular momentum (ties: higher shell index);
// the Rys horizontal transfer moves momentum from the first to the second.
// Each pair owns a run of primitive pairs with the Gaussian-product data.
#pragma once
#include <stdint.h>

namespace pqb {

constexpr int kMaxL = 2;                         // shells up to d (cartesian)
constexpr int kNumPairClass = 6;                 // ss ps pp ds dp dd
constexpr int kNumQuartetClass = 21;             // bra class >= ket class

// Per-item screening of the direct builds (all fields optional):
//   molmask: batched bases, molecule m's items are skipped when molmask[m] == 0;
//   dmax:    per shell, a bound on |D_ij| over the shell's rows i (within
//            its molecule's block); an item (ab|cd) is skipped when
//            Q_ab Q_cd max(dmax[a], dmax[b], dmax[c], dmax[d]) < tau, Q the
//            Schwarz factors (the incremental builds of a batched SCF digest
//            density differences, most of which are small);
// and where their sums go:
//   cmask, cstride: block b adds to the copy b & cmask of Jacc and Kacc, cstride
//            numbers apart (0: there is one).
struct ItemScreen {
    const int *molmask;
    const double *dmax;
    const double *Qpair;
    double tau;
    int cmask;
    int cstride;
};

struct PairInfo {
    double A[3];       // centre of the first shell
    double AB[3];      // A - B
    int prim_off;      // first PrimPair
    int nprim;         // number of (screened) primitive pairs
    int fa, fb;        // first basis-function index of each shell
    int sa, sb;        // shell indices
    int cls;           // pair class: index of (La, Lb) in ss ps pp ds dp dd
    int la, lb;
    int nm;            // functions of the pair's molecule (batched bases; else nbf)
    int mol;           // the pair's molecule (batched bases; else 0)
    long long bo;      // D/J/K element (i, j) of the molecule is at bo + i*nm + j
                       // (global function indices; 0 for a single molecule)
};

// 96 bytes, 32-byte aligned.  The FP64 kernels fetch the Fock-build fields
// with one 256-bit and one 128-bit load; the FP32 kernels (mixed precision)
// fetch their single-precision copy, f[], with one 256-bit load.
struct __align__(32) PrimPair {
    double zeta;       // alpha_a + alpha_b
    double izeta;      // 1 / zeta (the recurrences multiply; no division per quartet)
    double P[3];       // Gaussian product centre
    double K;          // c_a c_b sqrt(2) pi^(5/4)/zeta exp(-alpha_a alpha_b/zeta |AB|^2)
    double alpha_a;    // exponent of the first shell's primitive (alpha_b = zeta - alpha_a)
    double pad_;
    float f[8];        // zeta, 1/zeta, P[3], K rounded to single precision, 0, 0
};

__host__ __device__ inline int pair_class(int la, int lb)   // la >= lb
{
    return la * (la + 1) / 2 + lb;
}

// Lists of whole quartets (packed integrals, Schwarz factors) hold items of up
// to 64^4 primitive quartets; in thread mode kCoopLanes lanes share one of more
// than kCoopItem.
constexpr int kCoopItem = 24, kCoopLanes = 8;

// Blocks for a grid-stride launch over n items, per_block at a time, `most` blocks
// at most.  In 64 bits: an int that counted the lanes of shared items would
// overflow from 2^28 of them (the (ss|ss) quartets of 216 contracted s shells).
__host__ __device__ constexpr int grid_blocks(int64_t n, int per_block, int most)
{
    return (n + per_block - 1) / per_block < most ? (int)((n + per_block - 1) / per_block) : most;
}

// Components of quartet class qc; classes of more than kThreadMax run in warp
// mode, in FP64 in both precision modes.
constexpr int kThreadMax = 81;

__host__ __device__ constexpr int pair_components(int c)   // ss ps pp ds dp dd
{
    return c == 0 ? 1 : (c == 1 ? 3 : (c == 2 ? 9 : (c == 3 ? 6 : (c == 4 ? 18 : 36))));
}

inline bool warp_class(int qc)
{
    int cb = 0;
    while ((cb + 1) * (cb + 2) / 2 <= qc) ++cb;
    return pair_components(cb) * pair_components(qc - cb * (cb + 1) / 2) > kThreadMax;
}

// quartet class index for bra class cb >= ket class ck
__host__ __device__ inline int quartet_class(int cb, int ck) { return cb * (cb + 1) / 2 + ck; }

}  // namespace pqb
