// FP64 tensor-core tiles: mma.m8n8k4 (tcgen05 has no FP64 kind) and the
// asynchronous copies that feed them.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace pqb {

// acc (8 x 8) += A (8 x 4) B (4 x 8).  Lane L holds A[L/4][L%4], B[L%4][L/4]
// and acc[L/4][2 (L%4)], acc[L/4][2 (L%4) + 1].
__device__ __forceinline__ void dmma(double (&acc)[2], double a, double b)
{
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(acc[0]), "+d"(acc[1])
                 : "d"(a), "d"(b));
}

// 8 bytes global -> shared, zeros when !ok (src must be a valid address either way)
__device__ __forceinline__ void cp_async8(double *dst, const double *src, bool ok)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
                 "l"(__cvta_generic_to_global(src)), "r"(ok ? 8 : 0)
                 : "memory");
}

// Up to two doubles, both addresses 16-byte aligned: the first `count` (0, 1
// or 2) from src, zeros for the rest.
__device__ __forceinline__ void cp_async16(double *dst, const double *src, int count)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
                 "l"(__cvta_generic_to_global(src)), "r"(8 * count)
                 : "memory");
}

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }

template <int N> __device__ __forceinline__ void cp_async_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

}  // namespace pqb
