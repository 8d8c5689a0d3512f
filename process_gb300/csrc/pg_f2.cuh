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

// exp(x) to about 1e-9 (0 below -104, x at most 88).  x = k ln 2 + y by a
// two-float product, then the Taylor series of exp(y), |y| <= 0.35: 1 + y +
// y^2 / 2 in two floats, the rest (below 0.008) in one.
__device__ __forceinline__ F2 f2_exp(F2 x) {
  if (!(x.h >= -104.f)) return {x.h != x.h ? x.h : 0.f, 0.f};
  const float k = rintf(__fmul_rn(x.h, 1.44269502f));
  constexpr float LN2_H = 0.693147182464599609f, LN2_L = -1.90465432e-09f;
  const float p = __fmul_rn(k, LN2_H), pe = __fmaf_rn(k, LN2_H, -p);
  F2 y = f2_sum(x.h, -p);
  y = f2_quick(y.h, __fadd_rn(y.l, __fsub_rn(__fmaf_rn(-k, LN2_L, x.l), pe)));
  const float q = __fmul_rn(y.h, y.h), qe = __fmaf_rn(y.h, y.h, -q);
  float t = __fmaf_rn(y.h, 1.f / 40320.f, 1.f / 5040.f);
  t = __fmaf_rn(t, y.h, 1.f / 720.f);
  t = __fmaf_rn(t, y.h, 1.f / 120.f);
  t = __fmaf_rn(t, y.h, 1.f / 24.f);
  t = __fmaf_rn(t, y.h, 1.f / 6.f);
  t = __fmul_rn(__fmul_rn(t, q), y.h);
  F2 r = f2_add({1.f, 0.f}, y);
  r = f2_add(r, f2_quick(__fmul_rn(0.5f, q), __fmaf_rn(0.5f, qe, __fmul_rn(y.h, y.l))));
  r = f2_add(r, {t, 0.f});
  const int e = int(k), e1 = e / 2;
  return f2_scale(f2_scale(r, pow2f(e1)), pow2f(e - e1));
}

// log2(x) to about 1e-9 absolute, x >= 0 (-inf at 0).  x = 2^e m, m in
// [sqrt(1/2), sqrt(2)); log(m) = 2 atanh((m - 1) / (m + 1)) as its odd power
// series: the first term in two floats, the rest (below 0.005) in one.
__device__ __forceinline__ F2 f2_log2(F2 x) {
  if (!(x.h > 0.f) || x.h > 3.4e38f) return {x.h == 0.f ? __int_as_float(int(0xff800000u)) : x.h, 0.f};
  int e = 0;
  if (x.h < 0x1p-60f) { x = f2_scale(x, 0x1p64f); e = -64; }
  const int d = (__float_as_int(x.h) - 0x3f3504f3) >> 23;
  e += d;
  const F2 m = f2_scale(f2_scale(x, pow2f(-(d / 2))), pow2f(-(d - d / 2)));
  const F2 t = f2_div(f2_quick(__fsub_rn(m.h, 1.f), m.l), f2_add(f2_sum(m.h, 1.f), {m.l, 0.f}));
  const float s = __fmul_rn(t.h, t.h);
  constexpr float C_H = 2.88539004325866699f, C_L = 3.85192598e-08f;   // 2 / ln 2
  float u = __fmaf_rn(s, 1.f / 11.f, 1.f / 9.f);
  u = __fmaf_rn(u, s, 1.f / 7.f);
  u = __fmaf_rn(u, s, 1.f / 5.f);
  u = __fmaf_rn(u, s, 1.f / 3.f);
  u = __fmul_rn(__fmul_rn(u, s), __fmul_rn(t.h, C_H));
  return f2_add({float(e), 0.f}, f2_add(f2_mul(t, {C_H, C_L}), {u, 0.f}));
}

}  // namespace pg
