// fp64_approx.cuh -- FP64 reciprocals, roots and quotients from the MUFU seeds.
//
// GB300 issues FP64 at 2 lanes per SM and cycle, so a division or square root
// of about ten FP64 instructions costs what ten pair terms' FMAs cost.  Here a
// seed y0 (rcp / rsqrt.approx.ftz.f64, 20 bits of mantissa: relative error e,
// |e| < 2^-19) takes one step of third order, from the series named at each,
// and quotients and roots one corrected product.  u = 2^-53 below; the bounds
// hold where nothing leaves the normal range, and everything else takes
// CUDA's own operator.  tests/test_gpu_fp64_ops.py holds all of them against
// CUDA's operators and against extended precision.
#ifndef G6_FP64_APPROX_CUH
#define G6_FP64_APPROX_CUH

#include <cuda_runtime.h>

namespace fp64 {

__device__ __forceinline__ bool mid_range(double x) {  // 2^-300 <= |x| < 2^300
  const unsigned e = (unsigned)__double2hiint(x) & 0x7ff00000u;
  return e - (723u << 20) < (600u << 20);
}
__device__ __forceinline__ bool mid_positive(double x) {  // 2^-300 <= x < 2^300
  return (unsigned)__double2hiint(x) - (723u << 20) < (600u << 20);
}

// 1/x: y + y (h + h^2), h = 1 - x y0 (the geometric series of 1 / (1 - h)).
// What the series leaves out is h^3 = e^3 < 2^-57; with the last rounding the
// error is below 1.07 u, an ulp: not the rounded reciprocal in every case.
__device__ __forceinline__ double rcp64(double x) {
  if (!mid_range(x)) return 1.0 / x;
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double h = __fma_rn(-x, y, 1.0);
  return __fma_rn(y, __fma_rn(h, h, h), y);
}

// 1/sqrt(x): y + y h (1/2 + 3/8 h), h = 1 - x y0^2 (the binomial series of
// (1 - h)^(-1/2)).  h is about 2 e, so 5/16 h^3 = 2.5 e^3 < 2^-55.7 is left
// out; x y0 is rounded (u / 2 of the result), the last FMA is (u): below 1.7 u.
// For x normal; rsqrt64 takes any x.
__device__ __forceinline__ double rsqrt64_normal(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double h = __fma_rn(-(x * y), y, 1.0);
  return __fma_rn(h * y, __fma_rn(0.375, h, 0.5), y);
}
__device__ __forceinline__ double rsqrt64(double x) {
  return mid_positive(x) ? rsqrt64_normal(x) : 1.0 / sqrt(x);
}

// sqrt(x): q = x rsqrt64(x) and one Heron step in residual form, q + (x - q^2)
// / (2 sqrt x) with rsqrt64(x) / 2 as the divisor's reciprocal.  q is within 3 u,
// so the value before the last rounding is within 16 u^2 of the root: the
// result is the rounded root unless that lies so near the middle of two
// doubles (2^-49 ulp).
__device__ __forceinline__ double sqrt64(double x) {
  if (!mid_positive(x)) return sqrt(x);
  const double y = rsqrt64(x), q = x * y;
  return __fma_rn(__fma_rn(-q, q, x), 0.5 * y, q);
}

// a / b from y near 1 / b: q = a y and its residual times y (Markstein 1990,
// IBM J. Res. Dev. 34).  With the correctly rounded y his theorem 3 gives the
// rounded quotient.  With rcp64's y (1.07 u) q is within 2.1 u and the value
// before the last rounding within 5 u^2 of the quotient: the rounded quotient
// unless that lies so near the middle of two doubles (2^-50 ulp).  3 FP64
// instructions for each further quotient by the same b.  Where a product could
// leave the normal range (a = 0 too), the division itself.
__device__ __forceinline__ double div_by(double a, double b, double y, bool bmid) {
  if (!(bmid && mid_range(a))) return __ddiv_rn(a, b);
  const double q = __dmul_rn(a, y);
  return __fma_rn(__fma_rn(-b, q, a), y, q);
}
// Quotients by one b: div_by with rcp64's y.
struct Div {
  double b, y;
  bool mid;
  __device__ __forceinline__ explicit Div(double d) : b(d), y(rcp64(d)), mid(mid_range(d)) {}
  __device__ __forceinline__ double operator()(double a) const { return div_by(a, b, y, mid); }
  __device__ __forceinline__ double inv() const {  // 1 / b
    return mid ? __fma_rn(__fma_rn(-b, y, 1.0), y, y) : y;
  }
};
__device__ __forceinline__ double div64(double a, double b) { return Div(b)(a); }

}  // namespace fp64

#endif
