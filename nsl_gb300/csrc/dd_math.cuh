// Double-double arithmetic (unevaluated sums hi + lo of two FP64 numbers) of the double-double operators: error-free
// transformations (Dekker 1971; Knuth, TAOCP vol. 2, 4.2.2), products by FMA.
#pragma once

#include <cuda_runtime.h>

namespace nslg {

struct dd {
    double hi, lo;
};

__device__ __forceinline__ dd two_sum(double a, double b) {
    const double s = a + b;
    const double bb = s - a;
    return {s, (a - (s - bb)) + (b - bb)};
}
__device__ __forceinline__ dd fast_two_sum(double a, double b) {  // |a| >= |b|
    const double s = a + b;
    return {s, b - (s - a)};
}
// a + b, both double-double (the sum of the high parts exactly, the low parts added in FP64, renormalised)
__device__ __forceinline__ dd dd_add(dd a, dd b) {
    dd s = two_sum(a.hi, b.hi);
    s.lo += a.lo + b.lo;
    return fast_two_sum(s.hi, s.lo);
}
__device__ __forceinline__ dd dd_neg(dd a) { return {-a.hi, -a.lo}; }
// a * b with b an FP64 number: the product of the high part exactly (FMA), the low part's in FP64
__device__ __forceinline__ dd dd_mul_d(dd a, double b) {
    const double p = a.hi * b;
    const double e = fma(a.hi, b, -p);
    return fast_two_sum(p, fma(a.lo, b, e));
}

struct ddc {
    dd re, im;
};
// (a_r + i a_i) * v with a FP64 complex, v double-double complex
__device__ __forceinline__ ddc cmul_d(double2 a, ddc v) {
    return {dd_add(dd_mul_d(v.re, a.x), dd_neg(dd_mul_d(v.im, a.y))), dd_add(dd_mul_d(v.im, a.x), dd_mul_d(v.re, a.y))};
}
// conj(a) * v
__device__ __forceinline__ ddc cmulc_d(double2 a, ddc v) {
    return {dd_add(dd_mul_d(v.re, a.x), dd_mul_d(v.im, a.y)), dd_add(dd_mul_d(v.im, a.x), dd_neg(dd_mul_d(v.re, a.y)))};
}

}  // namespace nslg
