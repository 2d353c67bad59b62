// Precision-overloaded math used by the cell models.  MB_FAST_FP32_MATH
// switches the float functions to the hardware approximations (ex2.approx /
// lg2.approx through __expf / __logf, rcp.approx through __fdividef).
//
// The double exponential, reciprocal and quotient are written here without
// branches.  The cell models are chains of them (ToRORd: about 70 exponentials
// and 100 quotients per cell step), and a call with a branch for its special
// cases ends the basic block, so the scheduler cannot overlap one with the
// next: with the CUDA library's forms the FP64 ToRORd kernel kept its pipe
// 18 % busy.  The kernels that use the double exponential fill its table first
// (exp_table_fill).
#pragma once
#include <cuda_runtime.h>
#include "mb_exp2_table.h"

// Device code compiled with and without MB_FAST_FP32_MATH lives in different
// inline namespaces, so the two translation units never share a definition.
#ifdef MB_FAST_FP32_MATH
#define MB_NS_BEGIN namespace mb { inline namespace fastf {
#else
#define MB_NS_BEGIN namespace mb { inline namespace accf {
#endif
#define MB_NS_END } }

MB_NS_BEGIN

// ---- double ----------------------------------------------------------------------

// 1 / x from the hardware's approximation y (about 20 bits) by one third-order
// Newton step: with e = 1 - x y, 1/x = y / (1 - e) = y (1 + e + e^2) + O(e^3 / x).
// x finite, not zero and not beyond about 1e307: the models' denominators
// are sums of positive terms, their exponentials bounded by mexp.
__device__ __forceinline__ double mrcp(double x) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

// a / b: the product with 1/b and one correction by the remainder.
__device__ __forceinline__ double mdiv(double a, double b) {
    const double y = mrcp(b), q = a * y;
    return fma(fma(-b, q, a), y, q);
}

// 2^(j/128) and the relative remainder of its rounding, per block; the value's
// exponent field is lowered by j / 128 so that adding n 2^13 = (128 k + j) 2^13 to its
// high word gives 2^(k + j/128).
__device__ __forceinline__ double2 *exp_table() {
    __shared__ double2 tab[MB_EXP2_ROWS];
    return tab;
}

__device__ const double2 exp2_rows[MB_EXP2_ROWS] = {MB_EXP2_TABLE};

// Every thread of the block calls it before the first mexp(double).
__device__ __forceinline__ void exp_table_fill() {
    double2 *t = exp_table();
    for (unsigned j = threadIdx.x; j < MB_EXP2_ROWS; j += blockDim.x) {
        const double2 e = exp2_rows[j];
        t[j] = make_double2(__hiloint2double(__double2hiint(e.x) - (int)(j << 13), __double2loint(e.x)), e.y);
    }
    __syncthreads();
}

// exp(x), table-driven (P. T. P. Tang, ACM TOMS 15(2), 1989): with n the
// integer nearest 128 x / ln 2, x = n ln2/128 + r, |r| <= ln2/256, exp(x) =
// 2^(n/128) (1 + r + r^2/2 + ... + r^5/120), n = 128 k + j; the first omitted
// term is below 6e-19.  Arguments beyond +-700 are taken as +-700 (1e304, far
// from every value a rate of the models can still tell from infinity, so no
// denominator overflows).  NaN gives NaN: a concentration that has left its range
// (the logarithm or root of a negative value) reaches V through exponentials
// alone.  Its test is on the scale's side, off the chain through r.
__device__ __forceinline__ double mexp(double x) {
    const int hi = __double2hiint(x);
    x = __hiloint2double(min(hi & 0x7fffffff, 0x4085e000) | (hi & (int)0x80000000), __double2loint(x));   // 700.0
    const double shift = 0x1.8p52;
    const double t = fma(x, 0x1.71547652b82fep+7, shift);      // 128 / ln 2
    const int n = __double2loint(t);
    const double nd = t - shift;
    const double r = fma(-nd, 0x1.a39ef35793c76p-40, fma(-nd, 0x1.62e42fee00000p-8, x));
    const double2 row = exp_table()[n & (MB_EXP2_ROWS - 1)];
    double q = fma(r, 1.0 / 120.0, 1.0 / 24.0);
    q = fma(q, r, 1.0 / 6.0);
    q = fma(q, r, 0.5);
    const double p = fma(r * r, q, r + row.y);
    const bool nan = (hi & 0x7fffffff) > 0x7ff00000;
    const double s = __hiloint2double(nan ? 0x7ff80000 : __double2hiint(row.x) + n * 8192, __double2loint(row.x));
    return fma(s, p, s);
}

__device__ __forceinline__ double mlog(double x) { return log(x); }
__device__ __forceinline__ double msqrt(double x) { return sqrt(x); }
__device__ __forceinline__ double mexpm1(double x) { return expm1(x); }

// ---- float -----------------------------------------------------------------------

#ifdef MB_FAST_FP32_MATH
__device__ __forceinline__ float mexp(float x) { return __expf(x); }
__device__ __forceinline__ float mlog(float x) { return __logf(x); }
__device__ __forceinline__ float mdiv(float a, float b) { return __fdividef(a, b); }
__device__ __forceinline__ float mrcp(float x) { return __fdividef(1.0f, x); }
#else
__device__ __forceinline__ float mexp(float x) { return expf(x); }
__device__ __forceinline__ float mlog(float x) { return logf(x); }
__device__ __forceinline__ float mdiv(float a, float b) { return a / b; }
__device__ __forceinline__ float mrcp(float x) { return 1.0f / x; }
#endif
__device__ __forceinline__ float msqrt(float x) { return sqrtf(x); }
__device__ __forceinline__ float mexpm1(float x) { return expm1f(x); }

// ---- either ----------------------------------------------------------------------

// 1 / (1 + exp(x))
template <typename T>
__device__ __forceinline__ T sigm(const T x) { return mrcp(T(1.0) + mexp(x)); }

template <typename T>
__device__ __forceinline__ T sq(T x) { return x * x; }

MB_NS_END

// x / c for a literal c: the product with the literal's reciprocal.
#define MB_OVER(x, c) ((x) * T(1.0 / (c)))
