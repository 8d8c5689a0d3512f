// Expected-VAF binomial-mixture likelihood of an alt/depth table and its
// adjoint, batched over replicates (no reference counterpart: ProCESS has no
// calibration path; this is the differentiable form of the sequencing output
// used to fit epoch rates, exposures and purity to observed VAFs).
//
// Model of replicate r with K epochs, J signatures S_j over C classes:
//   w_k      = softmax(theta_k)                   (exposures of epoch k)
//   M_k(c)   = sum_j w_kj S_j(c)
//   pi_k(c)  = exp(lr_k) L_k M_k(c) / Z,   Z = sum_k exp(lr_k) L_k
//   v_k      = sigmoid(rho) phi_k / 2              (expected VAF of epoch k)
//   NLL      = - sum_i log sum_k pi_k(c_i) v_k^a_i (1 - v_k)^(d_i - a_i)
// (the binomial coefficient, constant in the parameters, is left out).
// Parameters per replicate, in order: lr_0..K-1, theta_00..theta_K-1,J-1, rho.
//
// The kernel is k_calib, one CTA per segment: a replicate's sites are cut into
// equal segments of at most CALIB_SEG sites, smaller ones where that fills the
// GPU.  A CTA computes the per-site log-likelihoods and responsibilities in
// FP32 with the replicate's constants and mixture weights in registers and
// only the site class's signature row S(c) gathered from shared memory:
//   u_k = log pi'_k / pi'_r + a log v_k / v_r + (d - a) log (1 - v_k) / (1 - v_r)
//         (pi'_k = exp(lr_k) L_k / Z, r a reference epoch)
//   e_k = exp(u_k - max u),  q_k = M_k(c) e_k,  s = sum_k q_k
//   gamma_k = q_k / s,  log-likelihood = the reference's + max u + log s
// and reduces
//   G_k = sum_i gamma_ik,  A_k = sum gamma_ik a_i,  B_k = sum gamma_ik (d_i - a_i),
//   H_kj = sum_i gamma_ik S_j(c_i) / M_k(c_i) = sum_i e_ik S_j(c_i) / s_i,  NLL
// (H carries the class dependence of the exposure gradient, so no per-class
// bins are needed) with per-thread FP32 sums over the thread's sites in
// order, a fixed warp tree and a Neumaier-compensated sum over the warps.  A
// replicate's segments are then added in a fixed order (compensated) and the
// chain rule applied, optionally followed by an Adam step on the parameters.
// Every sum has a fixed order: results are deterministic.
//
// While all segments are resident together, one launch does it all: each CTA
// derives its replicate's constants and the one that finishes a replicate's
// last segment runs its epilogue.  An evaluation of 2e5 sites took 24.7 us with
// separate kernels (and 13 CTAs of 16384 sites), now 12.4.  Adam steps repeat
// inside that launch, each replicate going on when its sums are complete:
// 200 steps over 64 x 5e4 sites took 5.4 ms as a graph of three kernels a step,
// 3.3 ms now.  With more segments than that, the constants and the
// epilogues are launches of their own (in k_calib they keep a CTA's slot from
// the next segment): 512 x 1e5 sites in 150 us.
// Persistent CTAs with equal shares of all sites took 190 us there: they reach
// their reductions together instead of overlapping them.
#pragma once
#include <cstdint>

#include "pg_f2.cuh"
#include "pg_kernels.h"

namespace pg {

constexpr int CAL_THREADS = 256;
constexpr int CAL_WARPS = CAL_THREADS / 32;
constexpr uint32_t CAL_MAXK = 8, CAL_MAXJ = 8, CAL_MAXC = 128;
constexpr uint32_t CAL_SPIN_LIMIT = 1u << 22;   // polls of a wait, 64 ns or more each

struct Neu {   // Neumaier-compensated FP32 sum
  float s = 0.f, c = 0.f;
  __device__ __forceinline__ void add(float x) {
    const float t = s + x;
    c += (fabsf(s) >= fabsf(x)) ? ((s - t) + x) : ((x - t) + s);
    s = t;
  }
  __device__ __forceinline__ float value() const { return s + c; }
  __device__ __forceinline__ float2 both() const {   // the value and what its rounding leaves
    const float v = s + c;
    return make_float2(v, (s - v) + c);
  }
};

// A replicate's parameters and constants in shared memory.  The site loop works
// on differences of log-likelihoods from those of a reference epoch (whose own
// sum over the sites is linear in the counts and added by the epilogue): for
// epoch k their constant, their slope in a and their slope in d, in base 2.
// The constants come from two-float arithmetic and are rounded together: what
// the slopes lose is put into the constant at the replicate's mean depth and
// the alt count expected of epoch k there, where its sites lie.  So the
// rounding of a constant, which every site shares, no longer adds up over the
// sites: the gradient of 512 tables of 1e5 sites is 2.0e-7 off (1.2e-6 with
// plain FP32 constants), 200 Adam steps over 64 tables of 5e4 sites, whose
// parameters keep their remainders too, typically 1.8e-6 (5e-6; up to 4e-5
// where Adam's oscillation amplifies rounding, now 2e-5).  It costs 1 to 2 us
// an evaluation.
template <uint32_t K, uint32_t J>
struct CalibRow {
  float p[K + K * J + 1], pl[K + K * J + 1], ew[K], phi[K];   // pl: the parameters' remainders (Adam steps)
  F2 logl[K];                            // log2 L_k
  F2 e[K + K * J + 1];                   // exponentials of the parameters (see calib_rows)
  float row[3 * K + 2 * K * J];          // constant, a, d (K each), the exposures w_kj (K x J) and their remainders
  float4 stat[2];                        // the replicate's sites and sums of a and of d - a (two floats each), its mean depth
  F2 c[K], lv[K], l1[K], odds[K];        // log2 exp(lr) L, log2 v, log2(1 - v), v / (1 - v)
  F2 prob[K];                            // pi_k = exp(lr_k) L_k / Z
  F2 logz;
  F2 lin[3];                             // the reference's log2 pi, log2 v, log2(1 - v)
  float v[K], sig;
};
template <uint32_t K, uint32_t J>
__device__ __forceinline__ void calib_load(CalibRow<K, J>& sh, const CalibArgs& a, const float* __restrict__ params,
                                           uint32_t r) {
  constexpr uint32_t P = K + K * J + 1;
  const uint32_t t = threadIdx.x;
  if (t < P) { sh.p[t] = __ldcg(params + uint64_t(r) * P + t); sh.pl[t] = 0.f; }
  else if (t >= 128 && t < 128 + K) sh.ew[t - 128] = a.epoch_w[r * K + t - 128];
  else if (t >= 160 && t < 160 + K) sh.phi[t - 160] = a.phi[r * K + t - 160];
  else if (t >= 176 && t < 176 + K) sh.logl[t - 176] = {a.epoch_log[r * K + t - 176].x, a.epoch_log[r * K + t - 176].y};
  else if (t >= 192 && t < 194) sh.stat[t - 192] = a.rep_stat[2 * r + t - 192];
  __syncthreads();
}
// One thread per function value and one copy of each function's code, loops
// rolled: the code runs once per evaluation, from far caches (unrolled per
// epoch and exposure it took 4.5 us longer).
template <uint32_t K, uint32_t J>
__device__ __forceinline__ void calib_rows(CalibRow<K, J>& sh) {
  constexpr uint32_t P = K + K * J + 1;
  constexpr F2 LOG2E = {1.44269502162933350f, 1.92596299e-08f}, one = {1.f, 0.f};
  const uint32_t t = threadIdx.x;
  auto par = [&](uint32_t q) { return F2{sh.p[q], sh.pl[q]}; };
  // x - m (infinite, or of equal infinities, as in FP32)
  auto less = [](F2 x, F2 m) {
    const float d = x.h == m.h ? 0.f : __fsub_rn(x.h, m.h);
    return fabsf(d) < 1e30f && fabsf(x.h) < 1e30f ? f2_add(x, f2_neg(m)) : F2{d, 0.f};
  };
  auto top = [&](uint32_t first, uint32_t n) {
    uint32_t m = first;
#pragma unroll 1
    for (uint32_t q = 1; q < n; ++q) m = sh.p[first + q] > sh.p[m] ? first + q : m;
    return par(m);
  };
  // exp(lr_k - max lr), exp(theta_kj - max theta_k) (probabilities do not depend
  // on a common term), exp(-|rho|)
  if (t < P) {
    F2 x = sh.p[t] >= 0.f ? f2_neg(par(t)) : par(t);
    if (t < P - 1) {
      const uint32_t first = t < K ? 0u : K + (t - K) / J * J;
      x = less(par(t), top(first, t < K ? K : J));
    }
    sh.e[t] = f2_exp(x);
  }
  __syncthreads();
  auto part = [&](uint32_t k) { return f2_mul(sh.e[k], {sh.ew[k], 0.f}); };
  auto total = [&]() {
    F2 z = {0.f, 0.f};
#pragma unroll 1
    for (uint32_t q = 0; q < K; ++q) z = f2_add(z, part(q));
    return z;
  };
  if (t < 2 * K + 1) {                   // log2 v_k, log2(1 - v_k), log2 Z
    const uint32_t k = t / 2;
    F2 x;
    if (t == 2 * K) {
      x = total();
    } else {
      const F2 e = sh.e[P - 1], sig = f2_div(sh.p[P - 1] >= 0.f ? one : e, f2_add(one, e));
      const F2 v = f2_mul(sig, {sh.phi[k] * 0.5f, 0.f}), w = f2_add(one, f2_neg(v));
      x = t & 1u ? w : v;
      if (t & 1u) sh.odds[k] = f2_div(v, w);
      else sh.v[k] = v.h;
      if (t == 0) sh.sig = sig.h;
    }
    const F2 y = f2_log2(x);
    (t == 2 * K ? sh.logz : t & 1u ? sh.l1[k] : sh.lv[k]) = y;
  } else if (t >= 32 && t < 32 + K * J) {
    const uint32_t x = t - 32;
    F2 den = {0.f, 0.f};
#pragma unroll 1
    for (uint32_t j = 0; j < J; ++j) den = f2_add(den, sh.e[K + x / J * J + j]);
    const F2 w = f2_div(sh.e[K + x], den);
    sh.row[3 * K + x] = w.h;
    sh.row[3 * K + K * J + x] = w.l;
  } else if (t >= 96 && t < 96 + K) {
    const uint32_t k = t - 96;
    sh.prob[k] = f2_div(part(k), total());
    const F2 x = less(par(k), top(0, K));
    sh.c[k] = x.h > -1e30f ? f2_add(f2_mul(x, LOG2E), sh.logl[k]) : F2{x.h, 0.f};
  }
  __syncthreads();
  if (t < K) {
    uint32_t best = 0;
#pragma unroll 1
    for (uint32_t q = 1; q < K; ++q)
      if (sh.c[q].h > sh.c[best].h) best = q;
    // the reference: a middle epoch, unless its share is negligible
    const uint32_t ref = sh.c[(K - 1) / 2].h >= sh.c[best].h - 30.f ? (K - 1) / 2 : best;
    const F2 l1r = sh.l1[ref], cr = sh.c[ref];
    const F2 d = f2_add(sh.l1[t], f2_neg(l1r));
    const F2 a = f2_add(f2_add(sh.lv[t], f2_neg(sh.lv[ref])), f2_neg(d));
    const F2 c = sh.c[t].h > -1e30f ? f2_add(sh.c[t], f2_neg(cr)) : sh.c[t];
    const float md = sh.stat[1].z, ma = md * sh.v[t];
    sh.row[t] = t == ref ? 0.f : c.h + (c.l + __fmaf_rn(ma, a.l, md * d.l));
    sh.row[K + t] = t == ref ? 0.f : a.h;
    sh.row[2 * K + t] = t == ref ? 0.f : d.h;
    if (t == 0) {
      sh.lin[0] = f2_add(cr, f2_neg(sh.logz));
      sh.lin[1] = sh.lv[ref];
      sh.lin[2] = l1r;
    }
  }
  __syncthreads();
}
template <uint32_t K, uint32_t J>
__device__ __forceinline__ void calib_tables(CalibRow<K, J>& sh, const CalibArgs& a, const float* __restrict__ params,
                                             uint32_t r) {
  calib_load<K, J>(sh, a, params, r);
  calib_rows<K, J>(sh);
}

// Per-site work: every thread takes sites i0 + tid, i0 + tid + 256, ...
// (coalesced, four sites' loads in flight at a time) and keeps plain FP32
// sums over its sites, in site order.  The signature rows in shared memory
// are JP floats (J rounded up to 4 or 8, zero beyond J).
// packed f32x2 arithmetic (two lanes of one 64-bit register pair, each
// rounded as the scalar operation)
__device__ __forceinline__ float2 f2fma(float2 a, float2 b, float2 c) {
  float2 d;
  asm("{\n\t.reg .b64 ra, rb, rc, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\tmov.b64 rc, {%6, %7};\n\t"
      "fma.rn.f32x2 rd, ra, rb, rc;\n\tmov.b64 {%0, %1}, rd;\n\t}"
      : "=f"(d.x), "=f"(d.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return d;
}
// four values read once: not kept in L1
__device__ __forceinline__ int4 load4(const int4* p) {
  int4 v;
  asm("ld.global.nc.L1::no_allocate.v4.s32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
  return v;
}
// base-2 exponential and logarithm (the PTX approximate instructions, FTZ)
__device__ __forceinline__ float ex2_approx(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float lg2_approx(float x) {
  float y;
  asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
#define PG_F2OP(NAME, OP)                                                                                        \
  __device__ __forceinline__ float2 NAME(float2 a, float2 b) {                                                \
    float2 d;                                                                                                  \
    asm("{\n\t.reg .b64 ra, rb, rd;\n\tmov.b64 ra, {%2, %3};\n\tmov.b64 rb, {%4, %5};\n\t" OP " rd, ra, rb;\n\t" \
        "mov.b64 {%0, %1}, rd;\n\t}"                                                                          \
        : "=f"(d.x), "=f"(d.y)                                                                                 \
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));                                                             \
    return d;                                                                                                  \
  }
PG_F2OP(f2mul, "mul.rn.f32x2")
PG_F2OP(f2add, "add.rn.f32x2")
#undef PG_F2OP

// CTAs per SM asked of the register allocator: the per-thread constants and
// sums take about 1 + 6K + 2KJ registers, plus K of per-site temporaries
// (4 CTAs, 64 registers, for the small shapes whose sums fit: 5% faster at
// K = 4, J = 3 than 3 CTAs)
constexpr uint32_t calib_min_blocks(uint32_t K, uint32_t J) {
  return (K + K % 2) * (J + 4) <= 28 && J <= 7 ? 4
         : 1 + 7 * K + 2 * K * J <= 53        ? 3
         : 1 + 7 * K + 2 * K * J <= 96        ? 2
                                              : 1;
}

// sum of v[x] over the warp for x < N (N <= 32): lane x ends with the sum of
// v[x].  Each step sends the half of the values the partner keeps: 31
// shuffles for 32 values instead of 160.
template <uint32_t N>
__device__ __forceinline__ float warp_transpose_sum(const float* v, uint32_t lane) {
  float w[32];
#pragma unroll
  for (uint32_t x = 0; x < 32; ++x) w[x] = x < N ? v[x] : 0.f;
#pragma unroll
  for (uint32_t h = 16; h >= 1; h >>= 1) {
    const bool up = (lane & h) != 0;
#pragma unroll
    for (uint32_t x = 0; x < h; ++x) {
      if (x >= N) continue;                 // both halves are padding
      const float send = up ? w[x] : w[x + h], keep = up ? w[x + h] : w[x];
      w[x] = keep + __shfl_xor_sync(0xffffffffu, send, h);
    }
  }
  return w[0];
}

// a replicate's segment sums -> NLL (tot[0]) and gradient
struct CalibEpilogue {
  float grp[CAL_THREADS / 32][1 + 3 * CAL_MAXK + CAL_MAXK * CAL_MAXJ][2];
  float2 tot[1 + 3 * CAL_MAXK + CAL_MAXK * CAL_MAXJ];
  float grad[CAL_MAXK + CAL_MAXK * CAL_MAXJ + 1], nll;
};
template <uint32_t K, uint32_t J>
__device__ __forceinline__ void calib_gradient(CalibEpilogue& sh, const CalibRow<K, J>& c, const CalibArgs& a,
                                               uint32_t r, const float2* partial) {
  constexpr uint32_t NV = 1 + 3 * K + K * J;
  const uint32_t c0 = a.rep_first_seg[r], c1 = a.rep_first_seg[r + 1];
  // warp g takes segments c0 + g, c0 + g + 8, ..., a lane one value (or three);
  // then the warps' sums in order
  const uint32_t lane = threadIdx.x & 31u, g = threadIdx.x >> 5;
  for (uint32_t x = lane; x < NV; x += 32) {
    Neu t;
#pragma unroll 4
    for (uint32_t q = c0 + g; q < c1; q += CAL_WARPS) {
      const float2 y = __ldcg(partial + uint64_t(q) * a.part_stride + x);
      t.add(y.x);
      t.c += y.y;
    }
    sh.grp[g][x][0] = t.s;
    sh.grp[g][x][1] = t.c;
  }
  __syncthreads();
  for (uint32_t x = threadIdx.x; x < NV; x += CAL_THREADS) {
    Neu t;
    for (uint32_t w = 0; w < CAL_WARPS; ++w) { t.add(sh.grp[w][x][0]); t.c += sh.grp[w][x][1]; }
    sh.tot[x] = t.both();
  }
  __syncthreads();
  // the gradient is a difference of sums that nearly cancel: the sums keep the
  // remainders of their rounding, and products enter unrounded (fma)
  const float2* G = sh.tot + 1 + 2 * K;
  const float2* H = sh.tot + 1 + 3 * K;
  const F2 n = {c.stat[0].x, c.stat[0].y};
  // d/d lr_k = N pi_k - G_k
  if (threadIdx.x < K) {
    const uint32_t k = threadIdx.x;
    const F2 g = f2_add(f2_mul(n, c.prob[k]), {-G[k].x, -G[k].y});
    sh.grad[k] = g.h + g.l;
  }
  if (threadIdx.x == 32) {
    // d/d rho = -(1 - sigma) sum_k (A_k - B_k v_k / (1 - v_k))
    F2 acc = {0.f, 0.f};
#pragma unroll 1
    for (uint32_t k = 0; k < K; ++k) {
      const float2 A = sh.tot[1 + k], B = sh.tot[1 + K + k];
      acc = f2_add(acc, f2_add({A.x, A.y}, f2_neg(f2_mul({B.x, B.y}, c.odds[k]))));
    }
    sh.grad[K + K * J] = -(1.f - c.sig) * (acc.h + acc.l);
  }
  if (threadIdx.x == 33) {
    // the reference epoch's log-likelihood of all sites: N log pi + sum a log v + sum (d - a) log(1 - v)
    F2 l = {0.f, 0.f};
    const float2* sums = reinterpret_cast<const float2*>(c.stat);
#pragma unroll 1
    for (uint32_t i = 0; i < 3 && n.h > 0.f; ++i) l = f2_add(l, f2_mul({sums[i].x, sums[i].y}, c.lin[i]));
    l = f2_mul(l, {0.693147182464599609f, -1.90465432e-09f});
    const F2 x = f2_add({sh.tot[0].x, sh.tot[0].y}, f2_neg(l));
    sh.nll = x.h + x.l;
  }
  // d/d theta_kj = -w_kj (sum_i gamma_ik S_j(c_i) / M_k(c_i) - G_k) = -w_kj (H_kj - G_k)
  if (threadIdx.x >= 64 && threadIdx.x < 64 + K * J) {
    const uint32_t x = threadIdx.x - 64;
    sh.grad[K + x] = -c.row[3 * K + x] * ((H[x].x - G[x / J].x) + (H[x].y - G[x / J].y));
  }
  __syncthreads();
}

// The Adam step's bias corrections of step `step` (from 0) and its update
struct AdamBias { float m, v; };
__device__ __forceinline__ AdamBias adam_bias(const AdamArgs& adam, uint32_t step) {
  const float t = float(step + 1);
  return {1.f - powf(adam.beta1, t), 1.f - powf(adam.beta2, t)};
}
// (the change of the parameter, to be subtracted)
__device__ __forceinline__ float adam_update(const AdamArgs& adam, AdamBias b, float g, float& m, float& v) {
  m = adam.beta1 * m + (1.f - adam.beta1) * g;
  v = adam.beta2 * v + (1.f - adam.beta2) * g * g;
  const float mh = m / b.m, vh = v / b.v;
  return adam.lr * mh / (sqrtf(vh) + adam.eps);
}

// one evaluation's results (and Adam step), by one CTA per replicate
template <uint32_t K, uint32_t J>
__device__ __forceinline__ void calib_epilogue(CalibEpilogue& sh, const CalibRow<K, J>& c, const CalibArgs& a,
                                               float* __restrict__ params, uint32_t r, float* __restrict__ nll_out,
                                               float* __restrict__ grad_out, const AdamArgs& adam) {
  constexpr uint32_t P = K + K * J + 1;
  calib_gradient<K, J>(sh, c, a, r, a.partial);
  if (threadIdx.x == 0 && nll_out) nll_out[r] = sh.nll;
  for (uint32_t q = threadIdx.x; q < P; q += CAL_THREADS) {
    const uint64_t o = uint64_t(r) * P + q;
    const float gq = sh.grad[q];
    if (grad_out) grad_out[o] = gq;
    if (adam.m) {
      float m = __ldcg(adam.m + o), v = __ldcg(adam.v + o);
      params[o] = c.p[q] - adam_update(adam, adam_bias(adam, adam.t), gq, m, v);
      adam.m[o] = m; adam.v[o] = v;
    }
  }
}

// STEPS: a.steps Adam steps in a cooperative launch (an instance of its own: in
// the other the step's state would spill; with 64 registers it spills even so,
// 4.6 ms against 3.3 with one CTA per SM less).  Every CTA of a replicate keeps the
// parameters and moments and makes each step itself, from all the segments'
// sums in the same order, so a step has one wait (the sums) where parameters
// published by one CTA need a second: 0.4 ms of 200 steps over 64 x 5e4 sites.
// The sums alternate between two halves of a.partial: a CTA is at
// most one step ahead of the others.
template <uint32_t K, uint32_t J, bool STEPS>
__global__ void __launch_bounds__(CAL_THREADS, calib_min_blocks(K, J) - (STEPS && calib_min_blocks(K, J) > 3 ? 1 : 0)) k_calib(CalibArgs a, float* __restrict__ params,
                                                                               float* __restrict__ nll_out,
                                                                               float* __restrict__ grad_out,
                                                                               AdamArgs adam) {
  constexpr uint32_t JP = J > 4 ? 8 : 4;
  constexpr uint32_t NV = 1 + 3 * K + K * J;   // nll, A, B, G, H
  constexpr uint32_t TAB = 3 * K + 2 * K * J;
  // signature rows, eight copies of each 16 bytes: a lane reads the copy in its
  // own banks, so the gather is free of conflicts (one copy: 2.9 lanes a bank)
  // The mixtures M_k(c) likewise, by class.
  constexpr uint32_t KP = K > 4 ? 8 : 4;
  __shared__ float4 s_sig[JP / 4][CAL_MAXC * 8], s_mix[KP / 4][CAL_MAXC * 8];
  __shared__ CalibRow<K, J> s_c;
  __shared__ union { float red[CAL_WARPS][NV]; CalibEpilogue epi; } s_u;
  __shared__ uint32_t s_go;
  // STEPS: the moments of the parameters, the step's bias corrections
  __shared__ float s_adam[2][STEPS ? K + K * J + 1 : 1];
  __shared__ AdamBias s_bias;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t seg = a.seg0 + blockIdx.x, r = a.seg_rep[seg];
  const uint64_t i0 = a.seg_start[seg], i1 = i0 + a.seg_len[seg];
  if (STEPS) {
    if (threadIdx.x < K + K * J + 1) s_adam[0][threadIdx.x] = s_adam[1][threadIdx.x] = 0.f;
    calib_load<K, J>(s_c, a, params, r);
  }
  for (uint32_t step = 0;; ++step) {   // a.steps evaluations (STEPS), or one
  if (STEPS) {
    if (threadIdx.x == 128) s_bias = adam_bias(adam, step);
    calib_rows<K, J>(s_c);
  } else if (a.tab) {
    for (uint32_t x = threadIdx.x; x < TAB; x += CAL_THREADS) s_c.row[x] = a.tab[uint64_t(r) * TAB + x];
    __syncthreads();
  } else {
    calib_tables<K, J>(s_c, a, params, r);
  }
  const float* s_row = s_c.row;
  for (uint32_t x = threadIdx.x; x < a.C * 8; x += CAL_THREADS) {
    float sg[JP], m[KP];
#pragma unroll
    for (uint32_t j = 0; j < JP; j += 4) {
      float4 v;
      if (STEPS && step) {
        v = s_sig[j / 4][x];
      } else {
        v = __ldg(reinterpret_cast<const float4*>(a.sig_rows) + ((x >> 3) * JP + j) / 4);
        s_sig[j / 4][x] = v;
      }
      sg[j] = v.x; sg[j + 1] = v.y; sg[j + 2] = v.z; sg[j + 3] = v.w;
    }
#pragma unroll
    for (uint32_t k = 0; k < KP; ++k) {
      m[k] = 0.f;
      if (k < K) {
#pragma unroll
        for (uint32_t j = 0; j < J; ++j) m[k] = __fmaf_rn(s_row[3 * K + K * J + k * J + j], sg[j], m[k]);
#pragma unroll
        for (uint32_t j = 0; j < J; ++j) m[k] = __fmaf_rn(s_row[3 * K + k * J + j], sg[j], m[k]);
      }
    }
#pragma unroll
    for (uint32_t k = 0; k < KP; k += 4) s_mix[k / 4][x] = make_float4(m[k], m[k + 1], m[k + 2], m[k + 3]);
  }
  __syncthreads();
  // epochs in pairs (packed f32x2 arithmetic); an odd K gets a padding
  // epoch of weight exp(-inf) = 0
  constexpr uint32_t KH = (K + 1) / 2;
  float2 cst[KH], dlv[KH], l1v[KH];
  auto at = [&](uint32_t k, uint32_t off, float pad) { return k < K ? s_row[off + k] : pad; };
  // the log-domain terms are in base 2 (ex2 / lg2 directly, the NLL scaled back by ln 2)
  constexpr float LN2 = 0.6931471805599453f;
#pragma unroll
  for (uint32_t h = 0; h < KH; ++h) {
    cst[h] = make_float2(at(2 * h, 0, 0.f), at(2 * h + 1, 0, -INFINITY));
    // u_k = cst_k + a dlv_k + d l1v_k
    l1v[h] = make_float2(at(2 * h, 2 * K, 0.f), at(2 * h + 1, 2 * K, 0.f));
    dlv[h] = make_float2(at(2 * h, K, 0.f), at(2 * h + 1, K, 0.f));
  }
  float nll = 0.f;
  float2 A[KH], D[KH], G[KH], H[J][KH];   // D_k = sum gamma_ik d_i (B_k = D_k - A_k)
#pragma unroll
  for (uint32_t h = 0; h < KH; ++h) {
    A[h] = D[h] = G[h] = make_float2(0.f, 0.f);
#pragma unroll
    for (uint32_t j = 0; j < J; ++j) H[j][h] = make_float2(0.f, 0.f);
  }
  auto site = [&](float al, float dl, int32_t c) {
    const uint32_t row = uint32_t(c) * 8 + (threadIdx.x & 7u);
    float sg[JP];
#pragma unroll
    for (uint32_t j = 0; j < JP; j += 4) {
      const float4 x = s_sig[j / 4][row];
      sg[j] = x.x; sg[j + 1] = x.y; sg[j + 2] = x.z; sg[j + 3] = x.w;
    }
    float2 m[(KP + 1) / 2];
#pragma unroll
    for (uint32_t k = 0; k < KP; k += 4) {
      const float4 x = s_mix[k / 4][row];
      m[k / 2] = make_float2(x.x, x.y); m[k / 2 + 1] = make_float2(x.z, x.w);
    }
    const float2 al2 = make_float2(al, al), dl2 = make_float2(dl, dl);
    float2 u[KH];
    float umax = -INFINITY;
#pragma unroll
    for (uint32_t h = 0; h < KH; ++h) {
      u[h] = f2fma(dl2, l1v[h], f2fma(al2, dlv[h], cst[h]));
      umax = fmaxf(umax, fmaxf(u[h].x, u[h].y));
    }
    float2 e[KH], q[KH], s2;
    const float2 nmax = make_float2(-umax, -umax);
#pragma unroll
    for (uint32_t h = 0; h < KH; ++h) {
      const float2 z = f2add(u[h], nmax);
      e[h] = make_float2(ex2_approx(z.x), ex2_approx(z.y));
      q[h] = f2mul(m[h], e[h]);
      s2 = h ? f2add(s2, q[h]) : q[h];
    }
    // a class that no epoch's mixture can emit (every M_k(c) = 0) keeps a
    // finite, tiny sum
    const float sum = fmaxf(s2.x + s2.y, 1e-30f);
    const float inv = __fdividef(1.f, sum);
    nll -= umax + lg2_approx(sum);
    const float2 inv2 = make_float2(inv, inv);
#pragma unroll
    for (uint32_t h = 0; h < KH; ++h) {
      const float2 g = f2mul(q[h], inv2), r = f2mul(e[h], inv2);
      A[h] = f2fma(g, al2, A[h]);
      D[h] = f2fma(g, dl2, D[h]);
      G[h] = f2add(G[h], g);
#pragma unroll
      for (uint32_t j = 0; j < J; ++j) H[j][h] = f2fma(r, make_float2(sg[j], sg[j]), H[j][h]);
    }
  };
  auto site_at = [&](uint64_t x) { site(float(__ldg(a.alt + x)), float(__ldg(a.depth + x)), __ldg(a.cls + x)); };
  auto site4 = [&](const int4& x, const int4& y, const int4& z) {
    site(float(x.x), float(y.x), z.x); site(float(x.y), float(y.y), z.y);
    site(float(x.z), float(y.z), z.z); site(float(x.w), float(y.w), z.w);
  };
  {
    // four consecutive sites per 16-byte load of each column (the columns
    // are 16-byte aligned); the unaligned head [i0, v0) and tail [v1, i1)
    // (under four sites each) site by site
    const uint64_t v0 = min((i0 + 3) & ~uint64_t(3), i1), v1 = max(i1 & ~uint64_t(3), v0);
    if (threadIdx.x < v0 - i0) site_at(i0 + threadIdx.x);
    if (threadIdx.x < i1 - v1) site_at(v1 + threadIdx.x);
    const int4* a4 = reinterpret_cast<const int4*>(a.alt) + v0 / 4;
    const int4* d4 = reinterpret_cast<const int4*>(a.depth) + v0 / 4;
    const int4* c4 = reinterpret_cast<const int4*>(a.cls) + v0 / 4;
    const uint32_t n4 = uint32_t((v1 - v0) / 4);
    // unrolled by three for the small shapes: 148 us for 512 x 1e5 sites (one
    // group a turn 165, two 153, four 164: spills)
#pragma unroll (K * J <= 16 ? 3 : 1)
    for (uint32_t q = threadIdx.x; q < n4; q += CAL_THREADS) site4(load4(a4 + q), load4(d4 + q), load4(c4 + q));
  }
  // block partial: warp trees, then a compensated sum over the warps
  float acc[NV];
  acc[0] = nll * LN2;
#pragma unroll
  for (uint32_t k = 0; k < K; ++k) {
    const bool hi = k & 1;
    acc[1 + k] = hi ? A[k / 2].y : A[k / 2].x;
    acc[1 + K + k] = hi ? D[k / 2].y - A[k / 2].y : D[k / 2].x - A[k / 2].x;
    acc[1 + 2 * K + k] = hi ? G[k / 2].y : G[k / 2].x;
#pragma unroll
    for (uint32_t j = 0; j < J; ++j) acc[1 + 3 * K + k * J + j] = hi ? H[j][k / 2].y : H[j][k / 2].x;
  }
#pragma unroll
  for (uint32_t q = 0; q < NV; q += 32) {
    constexpr uint32_t tail = NV % 32 ? NV % 32 : 32;
    const float v = q + 32 <= NV ? warp_transpose_sum<32>(acc + q, lane) : warp_transpose_sum<tail>(acc + q, lane);
    if (q + lane < NV) s_u.red[warp][q + lane] = v;
  }
  __syncthreads();
  // segment sums: nll, A_k, B_k, G_k, H_kj (j < J)
  float2* const sums = STEPS && (step & 1u) ? a.partial + uint64_t(gridDim.x) * a.part_stride : a.partial;
  float2* out = sums + uint64_t(seg) * a.part_stride;
  for (uint32_t x = threadIdx.x; x < NV; x += CAL_THREADS) {
    Neu t;
    for (uint32_t w = 0; w < CAL_WARPS; ++w) t.add(s_u.red[w][x]);
    out[x] = t.both();
  }
  if (!STEPS && a.tab) return;
  __threadfence();
  __syncthreads();
  const uint32_t n = a.rep_first_seg[r + 1] - a.rep_first_seg[r];
  if constexpr (!STEPS) {
    // the CTA that finishes the replicate's last segment runs the epilogue (the
    // count is left at zero for the next evaluation)
    if (threadIdx.x == 0) {
      s_go = atomicAdd(a.rep_done + r, 1u) + 1u == n ? 1u : 0u;
      if (s_go) a.rep_done[r] = 0u;
      __threadfence();
    }
    __syncthreads();
    if (s_go) calib_epilogue<K, J>(s_u.epi, s_c, a, params, r, nll_out, grad_out, adam);
    return;
  } else {
    constexpr uint32_t P = K + K * J + 1;
    // All the replicate's sums of this step.  The CTAs are all resident (a
    // cooperative launch); a wait that runs out all the same marks the call and
    // every CTA leaves at its next look.
    if (threadIdx.x == 0) {
      uint32_t go = 1, polls = 0;
      atomicAdd(a.rep_done + r, 1u);
      while (*reinterpret_cast<volatile uint32_t*>(a.rep_done + r) < (step + 1) * n) {
        if (++polls > CAL_SPIN_LIMIT || *reinterpret_cast<volatile uint32_t*>(a.status)) { go = 0; break; }
        __nanosleep(20);
      }
      __threadfence();
      if (!go) atomicExch(a.status, 1u);
      s_go = go;
    }
    __syncthreads();
    const bool first = seg == a.rep_first_seg[r];
    if (!s_go) {
      if (threadIdx.x == 0) {                    // no result: NaN
        params[uint64_t(r) * P] = __int_as_float(0x7fc00000);
        if (nll_out) nll_out[r] = __int_as_float(0x7fc00000);
      }
      return;
    }
    calib_gradient<K, J>(s_u.epi, s_c, a, r, sums);
    const bool end = step + 1 == a.steps;
    if (threadIdx.x < P) {
      const float u = adam_update(adam, s_bias, s_u.epi.grad[threadIdx.x], s_adam[0][threadIdx.x], s_adam[1][threadIdx.x]);
      const F2 p = f2_add({s_c.p[threadIdx.x], s_c.pl[threadIdx.x]}, {-u, 0.f});
      s_c.p[threadIdx.x] = p.h;
      s_c.pl[threadIdx.x] = p.l;
      if (end && first) params[uint64_t(r) * P + threadIdx.x] = p.h;
    }
    if (end) {
      if (first && threadIdx.x == 0 && nll_out) nll_out[r] = s_u.epi.nll;
      return;
    }
    __syncthreads();
  }
  }
}

// The constants and the epilogues in launches of their own, one CTA per
// replicate (see calib_launch)
template <uint32_t K, uint32_t J>
__global__ void __launch_bounds__(CAL_THREADS) k_calib_tables(CalibArgs a, const float* __restrict__ params) {
  __shared__ CalibRow<K, J> s_c;
  const uint32_t r = a.rep0 + blockIdx.x;
  calib_tables<K, J>(s_c, a, params, r);
  constexpr uint32_t TAB = 3 * K + 2 * K * J;
  for (uint32_t x = threadIdx.x; x < TAB; x += CAL_THREADS) a.tab[uint64_t(r) * TAB + x] = s_c.row[x];
}
template <uint32_t K, uint32_t J>
__global__ void __launch_bounds__(CAL_THREADS) k_calib_epilogue(CalibArgs a, float* __restrict__ params,
                                                                float* __restrict__ nll_out,
                                                                float* __restrict__ grad_out, AdamArgs adam) {
  __shared__ CalibRow<K, J> s_c;
  __shared__ CalibEpilogue s_epi;
  const uint32_t r = a.rep0 + blockIdx.x;
  calib_tables<K, J>(s_c, a, params, r);
  calib_epilogue<K, J>(s_epi, s_c, a, params, r, nll_out, grad_out, adam);
}

template <uint32_t K, uint32_t J>
static void calib_run(const CalibArgs& a, uint32_t n_segs, uint32_t n_rep, float* params, float* nll, float* grad,
                      const AdamArgs& adam, cudaStream_t st) {
  if (a.tab) k_calib_tables<K, J><<<n_rep, CAL_THREADS, 0, st>>>(a, params);
  if (a.steps == 1) {
    k_calib<K, J, false><<<n_segs, CAL_THREADS, 0, st>>>(a, params, nll, grad, adam);
  } else {
    CalibArgs aa = a;
    AdamArgs ad = adam;
    void* args[] = {&aa, &params, &nll, &grad, &ad};
    cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(k_calib<K, J, true>), dim3(n_segs), dim3(CAL_THREADS), args, 0, st);
  }
  if (a.tab) k_calib_epilogue<K, J><<<n_rep, CAL_THREADS, 0, st>>>(a, params, nll, grad, adam);
  note_launch(a.tab ? 3 : 1);
}

template <uint32_t K, uint32_t J>
static int calib_resident() {
  int n = 0, m = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k_calib<K, J, false>, CAL_THREADS, 0) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&m, k_calib<K, J, true>, CAL_THREADS, 0) != cudaSuccess)
    return 1;
  n = n < m ? n : m;
  return n > 0 ? n : 1;
}

#define PG_CALIB_J(KK, JJ) case KK * 8 + JJ - 9: PG_CALIB_DO(KK, JJ); break;
#define PG_CALIB_K(KK) PG_CALIB_J(KK, 1) PG_CALIB_J(KK, 2) PG_CALIB_J(KK, 3) PG_CALIB_J(KK, 4) \
                       PG_CALIB_J(KK, 5) PG_CALIB_J(KK, 6) PG_CALIB_J(KK, 7) PG_CALIB_J(KK, 8)

// the launcher and the residency of the shapes with at most four epochs and
// with more, in translation units of their own (they compile in parallel)
void calib_launch_lo(const CalibArgs& a, uint32_t n_segs, uint32_t n_rep, float* params, float* nll, float* grad,
                     const AdamArgs& adam, cudaStream_t st);
void calib_launch_hi(const CalibArgs& a, uint32_t n_segs, uint32_t n_rep, float* params, float* nll, float* grad,
                     const AdamArgs& adam, cudaStream_t st);
int calib_ctas_lo(uint32_t K, uint32_t J);
int calib_ctas_hi(uint32_t K, uint32_t J);

}  // namespace pg
