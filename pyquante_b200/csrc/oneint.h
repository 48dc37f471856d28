// One-electron integrals and their gradient over a per-function table
// (kernels in oneint.cu).
#pragma once
#include <cuda_runtime.h>

namespace pqb {

// Per-function table: functions f with origin[3f..], powers[3f..] and the
// primitives [prim_off[f], prim_off[f+1]) of exps/cn; norms[f] multiplies.
struct FuncTable {
    const double *origin;
    const int *powers;
    const int *prim_off;
    const double *exps, *cn, *norms;
};

// S, Tk, V (n x n, any may be null) for atoms[4*natoms] = {x, y, z, Z} (read
// for V only).
cudaError_t launch_oneint(int n, const FuncTable &ft, int natoms, const double *atoms, double *S, double *Tk, double *V,
                          cudaStream_t st);
// Adds 2 tr(D d(T+V)) - 2 tr(W dS) to grad[3*natoms].
cudaError_t launch_oneint_grad(int n, const FuncTable &ft, int natoms, const double *atoms, const int *func_atom,
                               const double *D, const double *W, double *grad, cudaStream_t st, int nsm);

}  // namespace pqb
