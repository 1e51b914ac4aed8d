// pt_fp64.cuh -- FP64 operations in the forms this part runs fastest, with the same roundings.
#pragma once

namespace pt {

// Products, sums and differences in the form of a fused multiply-add, each rounded once as they are: the
// unit takes a warp's DFMA every 16 cycles, its DMUL or DADD every 19.  (Kernel arguments, so that the
// compiler does not turn them back.)
struct FmaForms {
    double zero = -0.0, one = 1.0, minus = -1.0;
    __device__ __forceinline__ double mul(double a, double b) const { return __fma_rn(a, b, zero); }
    __device__ __forceinline__ double add(double a, double b) const { return __fma_rn(b, one, a); }
    __device__ __forceinline__ double sub(double a, double b) const { return __fma_rn(b, minus, a); }
};

// b / d, correctly rounded, from r = 1 / d (Markstein, IBM J. Res. Dev. 34 (1990): a quotient within an ulp,
// corrected once with its exact residual and a correctly rounded reciprocal, is the rounded quotient; two
// corrections bring b r there).  Five dependent operations where a division takes nine.  For exponents that
// keep every intermediate a normal number: in_range(b, 800) and in_range(d, 100).
__device__ __forceinline__ bool in_range(double v, int bits) {  // 2^-bits <= |v| < 2^bits
    return ((unsigned)__double2hiint(v) >> 20 & 0x7ffu) - (unsigned)(1023 - bits) < 2u * (unsigned)bits;
}
__device__ __forceinline__ double quotient(double b, double d, double r) {
    double q = __dmul_rn(b, r);
    q = __fma_rn(__fma_rn(-d, q, b), r, q);
    return __fma_rn(__fma_rn(-d, q, b), r, q);
}

}  // namespace pt
