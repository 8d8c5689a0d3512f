// The binomial and Poisson samplers of pg_rng.cuh, decided in FP32.
//
// A draw is a chain of decisions (accept, reject, an integer part) on
// quantities that pg_rng.cuh evaluates in FP64.  GB300 issues an FP64 warp
// instruction every 67 cycles per scheduler (32.5 ns measured, whatever the
// active lanes), so a tree level of binomial draws took 25 us.  Here the same
// quantities are evaluated on the FP32 pipes: as unevaluated sums of two
// floats (relative error below 2^-43) where an integer part is taken, as plain
// floats where two numbers are compared.  Each decision has a margin that
// exceeds the error of both evaluations; outside the margins the FP64
// sampler takes the same decisions from the same Philox words, so the result
// is its result.  Inside a margin the functions return false and the caller
// draws with the FP64 sampler.  Measured over 3.1e7 draws in each of fourteen
// ranges (none decided otherwise): Poisson means 1e-6 to 0.1 6e-5 of the draws,
// inversion up to means of ten 4e-4 (Poisson) and 9e-4 (binomial), rejection 3e-4
// to 8e-4, 1.8e-3 for binomials of 2^24 to 2^32 trials (the floor's margin grows
// with them); 1e-2 within 0.01 of a mean of ten, and every half of 20.
#pragma once
#include "pg_f2.cuh"
#include "pg_rng.cuh"

namespace pg {

__device__ __forceinline__ F2 f2_sqrt(F2 a) {   // a.h > 0
  const float s = __fsqrt_rn(a.h);
  const float e = __fadd_rn(__fmaf_rn(-s, s, a.h), a.l);
  return f2_quick(s, __fdividef(e, __fadd_rn(s, s)));
}
__device__ __forceinline__ F2 f2_u32(uint32_t x) {
  return f2_sum(float(x & 0xffff0000u), float(x & 0xffffu));
}
// x < 2^54, times 2^-54
__device__ __forceinline__ F2 f2_u54(uint64_t x) {
  const F2 a = f2_sum(float(uint32_t(x >> 30)) * 0x1p-24f, float(uint32_t(x >> 15) & 0x7fffu) * 0x1p-39f);
  return f2_quick(a.h, __fadd_rn(a.l, float(uint32_t(x) & 0x7fffu) * 0x1p-54f));
}
// a positive normal double scaled to [1, 2), and its exponent
__device__ __forceinline__ F2 f2_mantissa(double x, int& e) {
  const uint64_t bits = uint64_t(__double_as_longlong(x));
  e = int(bits >> 52) & 0x7ff;
  const uint64_t m = (bits & 0x000fffffffffffffull) | 0x0010000000000000ull;
  return f2_quick(float(uint32_t(m >> 29)) * 0x1p-23f, float(uint32_t(m) & 0x1fffffffu) * 0x1p-52f);
}

// floor of x (|x| < 2^33) and the distance of x to the nearest integer
__device__ __forceinline__ int64_t f2_floor(F2 x, float& dist) {
  const float fh = floorf(x.h);
  const float r = __fadd_rn(__fsub_rn(x.h, fh), x.l);
  const float fr = floorf(r), f = __fsub_rn(r, fr);
  dist = fminf(f, 1.f - f);
  return int64_t(fh) + int64_t(int32_t(fr));
}

// log1p(y) - y without cancellation
__device__ __forceinline__ float log1p_less(float y) {
  if (fabsf(y) < 0.125f) {
    float s = -1.f / 10.f;
    s = __fmaf_rn(s, y, 1.f / 9.f);  s = __fmaf_rn(s, y, -1.f / 8.f); s = __fmaf_rn(s, y, 1.f / 7.f);
    s = __fmaf_rn(s, y, -1.f / 6.f); s = __fmaf_rn(s, y, 1.f / 5.f);  s = __fmaf_rn(s, y, -1.f / 4.f);
    s = __fmaf_rn(s, y, 1.f / 3.f);  s = __fmaf_rn(s, y, -0.5f);
    return s * y * y;
  }
  return log1pf(y) - y;
}

// the Stirling tail of log k! (pg_stirling_tail) in FP32
__device__ __forceinline__ float stirling_tail_f(float k) {
  if (k <= 9.f) {
    // log k! - ((k + 1/2) log(k + 1) - (k + 1) + log(2 pi) / 2), k = 0 .. 9
    constexpr float t[10] = {0.0810614668f, 0.041340696f, 0.0276779257f, 0.0207906721f, 0.0166446912f,
                             0.0138761288f, 0.0118967099f, 0.0104112653f, 0.00925546218f, 0.00833056343f};
    float r = t[0];
#pragma unroll
    for (int i = 1; i < 10; ++i) r = k >= float(i) ? t[i] : r;
    return r;
  }
  const float i1 = __fdividef(1.f, k + 1.f), i2 = i1 * i1;
  return (1.f / 12.f - (1.f / 360.f - i2 * (1.f / 1260.f)) * i2) * i1;
}

// One attempt's uniforms of the transformed-rejection samplers, as FP64 sees
// them: U = u01_open(x, y) - 1/2 and us = 1/2 - |U|, both exact in FP64
// (multiples of 2^-54; the sum inside u01_open rounds half to even) and taken
// here from the same integers into two floats (2^-43 relative, which the margins
// hold), and V = u01_open(z, w).  False when us is so small that two floats lose
// it.
__device__ __forceinline__ bool attempt_uniforms(const U4& r, F2& U, F2& us, float& V) {
  const uint64_t u = ((uint64_t(r.x) << 32) | r.y) >> 11;
  const uint64_t t = u >= (1ull << 52) ? 2 * (u + (u & 1)) : 2 * u + 1;   // u01 * 2^54
  const int64_t s = int64_t(t) - (int64_t(1) << 53);
  const uint64_t m = uint64_t(s < 0 ? -s : s), d = (uint64_t(1) << 53) - m;
  if (d < (uint64_t(1) << 24)) return false;
  U = f2_u54(m);
  if (s < 0) U = f2_neg(U);
  us = f2_u54(d);
  const uint64_t v = ((uint64_t(r.z) << 32) | r.w) >> 11;
  V = __fmaf_rn(float(uint32_t(v >> 32)), 0x1p-21f, (float(uint32_t(v)) + 0.5f) * 0x1p-53f);
  return true;
}

// Margins: an integer part is taken when x is further from an integer than
// max(2^-18, n 2^-40) (n bounds the magnitudes that enter: FP64 is off by at
// most n 2^-49, two floats by n 2^-43); compared floats differ by at least
// 1e-4 + 1e-5 |x| (their errors stay below 5e-5 + 3e-6 |x|).
__device__ __forceinline__ float floor_margin(float n) { return fmaxf(0x1p-18f, n * 0x1p-40f); }
// a <= b: 1, a > b: 0, too close: -1
__device__ __forceinline__ int at_most(float a, float b, float margin) {
  const float d = a - b;
  return fabsf(d) <= margin ? -1 : (d < 0.f ? 1 : 0);
}

// binomial(st, n, p) with p = pp (or 1 - pp when flip), 0 < pp <= 1/2,
// n > 0.  True: k holds binomial's result.
__device__ __forceinline__ bool binomial_fast(Stream st, uint32_t n, F2 pp, bool flip, uint64_t& k) {
  const F2 nd = f2_u32(n);
  const F2 np = f2_mul(nd, pp);
  if (fabsf(np.h - 10.f) < 1e-4f) return false;
  int64_t kk = -1;
  if (np.h < 10.f) {
    // BINV: u against the running pmf
    const U4 r = st.next();
    const uint64_t v = ((uint64_t(r.x) << 32) | r.y) >> 11;
    float u = __fmaf_rn(float(uint32_t(v >> 32)), 0x1p-21f, (float(uint32_t(v)) + 0.5f) * 0x1p-53f);
    const float s = __fdividef(pp.h, 1.f - pp.h), aa = (nd.h + 1.f) * s;
    float rr = expf(nd.h * log1pf(-pp.h));
    kk = 0;
    for (;;) {
      if (fabsf(u - rr) < 2e-5f) return false;
      if (!(u > rr) || kk >= int64_t(n)) break;
      u -= rr;
      ++kk;
      rr *= __fdividef(aa, float(kk)) - s;
    }
  } else {
    const F2 q = f2_add({1.f, 0.f}, f2_neg(pp));
    const F2 spq = f2_sqrt(f2_mul(np, q));
    const F2 b = f2_add({1.14999998f, 2.38418583e-08f}, f2_mul({2.52999997f, 2.86102289e-08f}, spq));
    const F2 a = f2_add(f2_add({-0.0873000026f, 2.57492072e-09f}, f2_mul({0.0248000007f, -7.12275516e-10f}, b)),
                        f2_mul({0.00999999978f, 2.23517413e-10f}, pp));
    const F2 c = f2_add(np, {0.5f, 0.f});
    const float vr = 0.92f - __fdividef(4.2f, b.h);
    const float margin = floor_margin(nd.h);
    for (int it = 0; it < 16; ++it) {
      F2 U, us;
      float V;
      if (!attempt_uniforms(st.next(), U, us, V)) return false;
      const F2 t = f2_add(f2_div(f2_scale(a, 2.f), us), b);
      const F2 off = f2_mul(t, U);
      if (fabsf(off.h) > nd.h + 64.f) continue;     // far outside [0, n]
      float dist;
      const int64_t kd = f2_floor(f2_add(off, c), dist);
      if (dist < margin) return false;
      if (kd < 0 || kd > int64_t(n)) continue;
      if (fabsf(us.h - 0.07f) < 1e-6f) return false;
      if (us.h >= 0.07f) {
        const int sq = at_most(V, vr, 1e-5f);
        if (sq < 0) return false;
        if (sq) { kk = kd; break; }
      }
      // the exact test: log(V alpha / (a / us^2 + b)) <= log f(kd) - log f(m),
      // f the pmf and m its mode (a neighbour of the mode would do: the pmf
      // is flat there).  With x = kd - m, y1 = x / (m + 1), y2 = -x / (n - m + 1)
      // and the Stirling form of log k!, the right side is
      //   -(m + 1/2) (log1p y1 - y1) - (n - m + 1/2) (log1p y2 - y2)
      //   + x / 2 (1 / (m + 1) - 1 / (n - m + 1)) - x log1p(delta) + tails,
      //   1 + delta = (kd + 1) q / ((n - kd + 1) p)
      const float alpha = (2.83f + __fdividef(5.1f, b.h)) * spq.h;
      const float lhs = logf(__fdividef(V * alpha, __fdividef(a.h, us.h * us.h) + b.h));
      float frac;
      const F2 n1p = f2_add(np, pp);
      const int64_t m = f2_floor(n1p, frac);
      const float nf = floorf(n1p.h);                                    // rest: (n + 1) p - m, below 1
      const float rest = __fadd_rn(__fadd_rn(float(int64_t(nf) - m), __fsub_rn(n1p.h, nf)), n1p.l);
      const float x = float(kd - m), m1 = float(m) + 1.f, nm1 = float(int64_t(n) - m) + 1.f;
      const float delta = __fdividef(x + (1.f - pp.h - rest), (float(int64_t(n) - kd) + 1.f) * pp.h);
      const float ub = -(m1 - 0.5f) * log1p_less(__fdividef(x, m1)) - (nm1 - 0.5f) * log1p_less(-__fdividef(x, nm1)) +
                       0.5f * x * (__fdividef(1.f, m1) - __fdividef(1.f, nm1)) - x * log1pf(delta) +
                       stirling_tail_f(float(m)) + stirling_tail_f(float(int64_t(n) - m)) -
                       stirling_tail_f(float(kd)) - stirling_tail_f(float(int64_t(n) - kd));
      const int acc = at_most(lhs, ub, 1e-4f + 1e-5f * fabsf(ub));
      if (acc < 0) return false;
      if (acc) { kk = kd; break; }
    }
    if (kk < 0) return false;
  }
  k = flip ? uint64_t(n) - uint64_t(kk) : uint64_t(kk);
  return true;
}

// poisson(st, lambda), lambda > 0 normal and below 2^30.  True: k holds its result.
__device__ __forceinline__ bool poisson_fast(Stream st, double lambda, uint64_t& k) {
  int e;
  const F2 man = f2_mantissa(lambda, e);
  e -= 1023;
  if (e > 29 || e < -60) return false;
  const F2 lam = f2_scale(man, pow2f(e));
  if (fabsf(lam.h - 10.f) < 1e-4f) return false;
  if (lam.h < 10.f) {
    const U4 r = st.next();
    const uint64_t v = ((uint64_t(r.x) << 32) | r.y) >> 11;
    const float u = __fmaf_rn(float(uint32_t(v >> 32)), 0x1p-21f, (float(uint32_t(v)) + 0.5f) * 0x1p-53f);
    float p = expf(-lam.h), F = p;
    uint32_t kk = 0;
    for (;;) {
      if (fabsf(u - F) < 2e-5f) return false;
      if (!(u > F)) break;
      if (++kk > 60) return false;
      p *= __fdividef(lam.h, float(kk));
      F += p;
    }
    k = kk;
    return true;
  }
  const F2 slam = f2_sqrt(lam);
  const F2 b = f2_add({0.930999994f, 5.72204595e-09f}, f2_mul({2.52999997f, 2.86102289e-08f}, slam));
  const F2 a = f2_add({-0.0590000004f, 3.57627872e-10f}, f2_mul({0.0248300005f, -4.75049e-10f}, b));
  const F2 c = f2_add(lam, {0.430000007f, -7.15255721e-09f});
  const float invalpha = 1.1239f + __fdividef(1.1328f, b.h - 3.4f);
  const float vr = 0.9277f - __fdividef(3.6224f, b.h - 2.f);
  const float margin = floor_margin(lam.h);
  for (int it = 0; it < 16; ++it) {
    F2 U, us;
    float V;
    if (!attempt_uniforms(st.next(), U, us, V)) return false;
    const F2 off = f2_mul(f2_add(f2_div(f2_scale(a, 2.f), us), b), U);
    const F2 xk = f2_add(off, c);
    if (!(fabsf(xk.h) < 0x1p31f)) return false;
    float dist;
    const int64_t kd = f2_floor(xk, dist);
    if (dist < margin + fabsf(off.h) * 0x1p-40f) return false;
    if (fabsf(us.h - 0.07f) < 1e-6f || fabsf(us.h - 0.013f) < 1e-6f) return false;
    if (us.h >= 0.07f) {
      const int sq = at_most(V, vr, 1e-5f);
      if (sq < 0) return false;
      if (sq) { k = uint64_t(kd); return true; }
    }
    if (kd < 0) continue;
    if (us.h < 0.013f) {
      const int below = at_most(V, us.h, 1e-6f);
      if (below < 0) return false;
      if (!below) continue;
    }
    // log(V invalpha / (a / us^2 + b)) <= -lambda + kd log lambda - log kd!;
    // for kd >= 10, with y = (kd - lambda) / kd, the right side is
    //   kd (log1p(-y) + y) - log(2 pi kd) / 2 - 1 / (12 kd) + 1 / (360 kd^3)
    const float lhs = logf(__fdividef(V * invalpha, __fdividef(a.h, us.h * us.h) + b.h));
    const float kf = float(kd);
    float rhs;
    if (kd >= 10) {
      const float d = __fsub_rn(__fsub_rn(kf, lam.h), lam.l) + float(kd - int64_t(kf));   // kd - lambda
      const float ik = __fdividef(1.f, kf);
      rhs = kf * log1p_less(-d * ik) - 0.5f * logf(6.2831853f * kf) - ik * (1.f / 12.f) +
            ik * ik * ik * (1.f / 360.f);
    } else {
      float lf = 0.f;                        // log kd!
      for (int i = 2; i <= int(kd); ++i) lf += logf(float(i));
      rhs = kf * logf(lam.h) - lam.h - lf;
    }
    const int acc = at_most(lhs, rhs, 1e-4f + 1e-5f * fabsf(rhs));
    if (acc < 0) return false;
    if (acc) { k = uint64_t(kd); return true; }
  }
  return false;
}

}  // namespace pg
