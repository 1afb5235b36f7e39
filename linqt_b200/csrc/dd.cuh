// Double-double arithmetic (unevaluated sums hi + lo of two FP64 numbers, about 106 bits),
// from the error-free transformations of Knuth and Dekker.  A dd value is a double2 (x = hi,
// y = lo).
#pragma once

#include <cuda_runtime.h>

namespace linqt {

// s + e = a + b exactly (Knuth's two-sum)
__device__ __forceinline__ void two_sum(double a, double b, double &s, double &e) {
  s = __dadd_rn(a, b);
  const double t = __dsub_rn(s, a);
  e = __dadd_rn(__dsub_rn(a, __dsub_rn(s, t)), __dsub_rn(b, t));
}

// a + b
__device__ __forceinline__ double2 dd_add(double2 a, double2 b) {
  double s, e;
  two_sum(a.x, b.x, s, e);
  e = __dadd_rn(e, __dadd_rn(a.y, b.y));
  const double h = __dadd_rn(s, e);
  return make_double2(h, __dsub_rn(e, __dsub_rn(h, s)));
}

// a * b
__device__ __forceinline__ double2 dd_mul(double2 a, double2 b) {
  const double p = __dmul_rn(a.x, b.x);
  const double e = __fma_rn(a.y, b.x, __fma_rn(a.x, b.y, __fma_rn(a.x, b.x, -p)));
  const double h = __dadd_rn(p, e);
  return make_double2(h, __dsub_rn(e, __dsub_rn(h, p)));
}
__device__ __forceinline__ double2 dd_scale(double2 a, double b) {
  const double p = __dmul_rn(a.x, b);
  const double e = __fma_rn(a.y, b, __fma_rn(a.x, b, -p));
  const double h = __dadd_rn(p, e);
  return make_double2(h, __dsub_rn(e, __dsub_rn(h, p)));
}
// a / b
__device__ __forceinline__ double2 dd_div(double2 a, double b) {
  const double q = a.x / b;
  const double r = __dadd_rn(__fma_rn(-q, b, a.x), a.y);
  const double t = r / b;
  const double h = __dadd_rn(q, t);
  return make_double2(h, __dsub_rn(t, __dsub_rn(h, q)));
}

// c += a * b, c a running sum whose low part is not renormalised (|lo| grows by one unit of
// hi per term; dd_norm at the end)
__device__ __forceinline__ void dd_fma(double2 a, double2 b, double2 &c) {
  const double p = __dmul_rn(a.x, b.x);
  double e = __fma_rn(a.x, b.x, -p);
  e = __fma_rn(a.x, b.y, e);
  e = __fma_rn(a.y, b.x, e);
  double s, t;
  two_sum(c.x, p, s, t);
  c.x = s;
  c.y = __dadd_rn(c.y, __dadd_rn(t, e));
}
// c += a, the same
__device__ __forceinline__ void dd_acc(double2 a, double2 &c) {
  double s, t;
  two_sum(c.x, a.x, s, t);
  c.x = s;
  c.y = __dadd_rn(c.y, __dadd_rn(t, a.y));
}
__device__ __forceinline__ double2 dd_norm(double2 a) {
  double s, e;
  two_sum(a.x, a.y, s, e);
  return make_double2(s, e);
}
__device__ __forceinline__ double2 dd_neg(double2 a) { return make_double2(-a.x, -a.y); }

}  // namespace linqt
