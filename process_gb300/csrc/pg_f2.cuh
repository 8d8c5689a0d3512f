// Arithmetic on unevaluated sums of two floats (relative error below 2^-43): T.
// J. Dekker, "A floating-point technique for extending the available
// precision", Numer. Math. 18, 1971; D. E. Knuth, TAOCP vol. 2, 4.2.2 (the
// error of a sum).  Rounded operations throughout, so that no compiler
// contracts them.
#pragma once
#include <cstdint>

namespace pg {

struct F2 { float h, l; };   // h + l, |l| at most half an ulp of h

__device__ __forceinline__ F2 f2_quick(float a, float b) {   // |a| >= |b|
  const float s = __fadd_rn(a, b);
  return {s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ F2 f2_sum(float a, float b) {
  const float s = __fadd_rn(a, b), bb = __fsub_rn(s, a);
  return {s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb))};
}
__device__ __forceinline__ F2 f2_add(F2 a, F2 b) {
  const F2 s = f2_sum(a.h, b.h), t = f2_sum(a.l, b.l);
  const F2 u = f2_quick(s.h, __fadd_rn(s.l, t.h));
  return f2_quick(u.h, __fadd_rn(u.l, t.l));
}
__device__ __forceinline__ F2 f2_neg(F2 a) { return {-a.h, -a.l}; }
__device__ __forceinline__ F2 f2_mul(F2 a, F2 b) {
  const float p = __fmul_rn(a.h, b.h);
  float e = __fmaf_rn(a.h, b.h, -p);
  e = __fmaf_rn(a.h, b.l, e);
  e = __fmaf_rn(a.l, b.h, e);
  return f2_quick(p, e);
}
__device__ __forceinline__ F2 f2_scale(F2 a, float p2) { return {__fmul_rn(a.h, p2), __fmul_rn(a.l, p2)}; }  // p2 a power of two
__device__ __forceinline__ F2 f2_div(F2 a, F2 b) {
  const float q = __fdividef(a.h, b.h);
  // a - q b, then one more quotient digit
  const float p = __fmul_rn(q, b.h), pe = __fmaf_rn(q, b.h, -p);
  const F2 r = f2_add(a, {-p, -__fmaf_rn(q, b.l, pe)});
  const float q2 = __fdividef(r.h, b.h);
  return f2_quick(q, q2);
}
__device__ __forceinline__ float pow2f(int e) { return __int_as_float((e + 127) << 23); }   // -126 <= e <= 127

}  // namespace pg
