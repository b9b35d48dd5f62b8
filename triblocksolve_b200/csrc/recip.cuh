/*
 * recip.cuh -- FP64 reciprocals without a branch, for the pivot chains of the
 * line factorizations (kernels_fast.cu, kernels_ref.cu).
 */
#ifndef TBS_RECIP_CUH
#define TBS_RECIP_CUH

#include <cuda_runtime.h>

namespace tbs {

/* |v| within 2^-e .. 2^e (not zero, not infinite, a number) */
__device__ __forceinline__ bool within_pow2(double v, int e) {
    return (unsigned)((__double2hiint(v) & 0x7fffffff) - ((1023 - e) << 20)) < (unsigned)(2 * e) << 20;
}

/* every bit of the significand set (no branch: it stands in the chain) */
__device__ __forceinline__ bool ones_significand(double d) {
    return ((__double2hiint(d) | ~0xfffff) & __double2loint(d)) == -1;
}

/* RN(1 / d) for d within 2^-1000 .. 2^1000 whose significand is not all ones.
 * Newton's iteration x += x (1 - d x) doubles the correct bits of the
 * hardware's approximation (about 20) twice, so x is 1 / d rounded, but where
 * that is close to a tie: |1 - d x| <= 2^-53 (1 + 2^-20).  The last step's
 * remainder is exact, and its result (1 / d) (1 - (1 - d x)^2) before the
 * rounding, 2^-106 from 1 / d at most; no reciprocal is that close to a tie
 * but that of 2^53 - 1 (P. Markstein, IBM J. Res. Dev. 34 (1990) 111-119).
 * Six dependent operations behind the approximation; the exceptions are
 * noted without a branch, which a pivot's chain feels more than they do
 * (100 lines of 256 cells: 161 us, 198 with one). */
__device__ __forceinline__ double rcp_newton(double d) {
    double x;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(x) : "d"(d));
#pragma unroll
    for (int k = 0; k < 3; ++k) x = fma(x, fma(-d, x, 1.0), x);
    return x;
}

/* whether rcp_newton may be off for d */
__device__ __forceinline__ bool rcp_exception(double d) {
    return (int)!within_pow2(d, 1000) | (int)ones_significand(d);
}

}  // namespace tbs

#endif /* TBS_RECIP_CUH */
