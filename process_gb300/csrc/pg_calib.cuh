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
// A replicate's sites are cut into chunks of CAL_CHUNK, whose 256 threads take
// four consecutive sites at a time.  Per site, in FP32, with the replicate's
// constants in registers and only the rows of the site's class (signatures
// S(c), mixtures M(c)) gathered from shared memory:
//   u_k = log pi'_k + a log v_k + (d - a) log (1 - v_k)  (pi'_k = exp(lr_k) L_k / Z)
//   e_k = exp(u_k - max u),  q_k = M_k(c) e_k,  s = sum_k q_k
//   gamma_k = q_k / s,  log-likelihood = max u + log s
// Reduced are
//   G_k = sum_i gamma_ik,  A_k = sum gamma_ik a_i,  B_k = sum gamma_ik (d_i - a_i),
//   H_kj = sum_i gamma_ik S_j(c_i) / M_k(c_i) = sum_i e_ik S_j(c_i) / s_i,  NLL
// (H carries the class dependence of the exposure gradient, so no per-class
// bins are needed): per thread in the order of its sites, a fixed warp tree,
// compensated (Neumaier) sums over a chunk's eight warps and over the chunks,
// then the chain rule and, for a calibration loop, an Adam step.  Every sum has
// a fixed order that depends on the replicate's sites alone (and where they lie
// on the grid of four), so a replicate's results have the same bits in any
// batch and on either path below.
// Adam needs that: where it oscillates around the optimum, it amplifies a
// gradient's rounding a thousandfold.
//
// While all chunks are resident together, one launch (k_calib) does it all:
// each CTA derives its replicate's constants, and the one that finishes a
// replicate's last sums runs its epilogue.  The warps of a chunk go to several
// CTAs where that fills the GPU (by_warps): a replicate's warps are dealt out in
// turn to its CTAs.  Adam steps repeat inside that launch, each replicate
// going on when its sums are complete.  With more chunks than that, a CTA takes
// a chunk, and the constants and the epilogues are launches of their own (in
// k_calib they keep a CTA's slot from the next chunk).  Against three kernels
// with a CTA per chunk, K = 4, J = 3: 2e5 sites 25.7 -> 16.5 us, 512 x 1e5 sites
// 166 -> 148, 200 Adam steps over 64 x 5e4 sites (a graph of 600 launches) 4.98
// -> 3.66 ms; no shape from K = J = 1 to 8 is slower at 20001 to 100 x 120001
// sites.  Bound by the serial sums (64 sites a thread) while the GPU is not
// filled, then by the instructions per site.
#pragma once
#include <cstdint>

#include "pg_kernels.h"
#include "pg_wait.h"

namespace pg {

constexpr int CAL_THREADS = 256;
constexpr int CAL_WARPS = CAL_THREADS / 32;
constexpr uint32_t CAL_MAXK = 8, CAL_MAXJ = 8, CAL_MAXC = 128;
constexpr uint32_t CAL_CHUNK = 16384;   // sites (per-thread FP32 sums of 256 in site order)
// the arrivals' count before the first step: it wraps at once, not only after
// 2^32 arrivals
constexpr uint32_t CAL_COUNT0 = 0xffffffffu;

struct Neu {   // Neumaier-compensated FP32 sum
  float s = 0.f, c = 0.f;
  __device__ __forceinline__ void add(float x) {
    const float t = s + x;
    c += (fabsf(s) >= fabsf(x)) ? ((s - t) + x) : ((x - t) + s);
    s = t;
  }
  __device__ __forceinline__ float value() const { return s + c; }
};

// A replicate's parameters and constants in shared memory, calib_row_floats of
// them (floats alone: the launches of the split form copy it whole)
template <uint32_t K, uint32_t J>
struct CalibRow {
  float p[K + K * J + 1], ew[K], phi[K];
  float logw[K];                         // log L_k
  float e[K + K * J];                    // exp(lr_k), exp(theta_kj - max theta_k)
  float row[3 * K + K * J];              // log pi'_k, log v_k, log(1 - v_k) (K each), the exposures w_kj (K x J)
  float v[K], sig, z;
};
constexpr uint32_t calib_row_floats(uint32_t K, uint32_t J) { return 9 * K + 3 * K * J + 3; }
template <uint32_t K, uint32_t J>
__device__ __forceinline__ void calib_load(CalibRow<K, J>& sh, const CalibArgs& a, const float* __restrict__ params,
                                           uint32_t r) {
  constexpr uint32_t P = K + K * J + 1;
  const uint32_t t = threadIdx.x;
  if (t < P) {
    sh.p[t] = __ldcg(params + uint64_t(r) * P + t);
  } else if (t >= 128 && t < 128 + K) {
    sh.ew[t - 128] = a.epoch_w[r * K + t - 128];
    sh.logw[t - 128] = logf(sh.ew[t - 128]);
  } else if (t >= 160 && t < 160 + K) {
    sh.phi[t - 160] = a.phi[r * K + t - 160];
  }
  __syncthreads();
}
// One thread per function value: the code runs once per evaluation.
template <uint32_t K, uint32_t J>
__device__ __forceinline__ void calib_rows(CalibRow<K, J>& sh) {
  constexpr uint32_t P = K + K * J + 1;
  const uint32_t t = threadIdx.x;
  if (t < K) {
    sh.e[t] = expf(sh.p[t]);
  } else if (t < P - 1) {
    const float* th = sh.p + K + (t - K) / J * J;
    float mx = th[0];
#pragma unroll 1
    for (uint32_t j = 1; j < J; ++j) mx = fmaxf(mx, th[j]);
    sh.e[t] = expf(sh.p[t] - mx);
  } else if (t >= 96 && t < 96 + 2 * K) {   // log v_k, log(1 - v_k)
    const uint32_t k = (t - 96) / 2;
    const float sig = 1.f / (1.f + expf(-sh.p[P - 1]));
    const float v = sig * sh.phi[k] * 0.5f;
    if (t & 1u) {
      sh.row[2 * K + k] = log1pf(-v);
    } else {
      sh.row[K + k] = logf(v);
      sh.v[k] = v;
      if (k == 0) sh.sig = sig;
    }
  }
  __syncthreads();
  if (t < K) {
    float z = 0.f;
#pragma unroll 1
    for (uint32_t q = 0; q < K; ++q) z += sh.e[q] * sh.ew[q];
    sh.row[t] = sh.p[t] + sh.logw[t] - logf(z);
    if (t == 0) sh.z = z;
  } else if (t >= 32 && t < 32 + K * J) {
    const uint32_t x = t - 32;
    float den = 0.f;
#pragma unroll 1
    for (uint32_t j = 0; j < J; ++j) den += sh.e[K + x / J * J + j];
    sh.row[3 * K + x] = sh.e[K + x] / den;
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

// the Adam steps' instance, whose loop keeps more: two at most (200 steps over
// 64 x 5e4 sites: 3.66 ms, with three CTAs 3.81, over 20 x 5e4 at K = J = 2 2.2
// against 3.3 ms: spills)
constexpr uint32_t calib_ctas(uint32_t K, uint32_t J, bool steps) {
  return steps && calib_min_blocks(K, J) > 2 ? 2 : calib_min_blocks(K, J);
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

// a replicate's sums -> NLL (tot[0]) and gradient
struct CalibEpilogue {
  float grp[CAL_WARPS][1 + 3 * CAL_MAXK + CAL_MAXK * CAL_MAXJ];
  float tot[1 + 3 * CAL_MAXK + CAL_MAXK * CAL_MAXJ];
  float grad[CAL_MAXK + CAL_MAXK * CAL_MAXJ + 1];
};
template <uint32_t K, uint32_t J>
__device__ __forceinline__ void calib_gradient(CalibEpilogue& sh, const CalibRow<K, J>& c, const CalibArgs& a,
                                               uint32_t r, const float* partial) {
  constexpr uint32_t NV = 1 + 3 * K + K * J;
  const uint32_t c0 = a.rep_first_chunk[r], c1 = a.rep_first_chunk[r + 1];
  const uint32_t x = threadIdx.x, lane = x & 31u, g = x >> 5;
  Neu t;                                 // thread x: value x over the chunks, in order
  if (a.by_warps) {
    // eight chunks at a time, a warp adding up the warps of one
    for (uint32_t q0 = c0; q0 < c1; q0 += CAL_WARPS) {
      if (q0 + g < c1)
        for (uint32_t y = lane; y < NV; y += 32) {
          const float* at = partial + uint64_t(q0 + g) * CAL_WARPS * a.part_stride + y;
          float f[CAL_WARPS];
#pragma unroll
          for (uint32_t w = 0; w < CAL_WARPS; ++w) f[w] = __ldcg(at + w * a.part_stride);
          Neu u;
#pragma unroll
          for (uint32_t w = 0; w < CAL_WARPS; ++w) u.add(f[w]);
          sh.grp[g][y] = u.value();
        }
      __syncthreads();
      if (x < NV)
        for (uint32_t q = 0; q < min(c1 - q0, uint32_t(CAL_WARPS)); ++q) t.add(sh.grp[q][x]);
      __syncthreads();
    }
  } else if (x < NV) {
#pragma unroll 8
    for (uint32_t q = c0; q < c1; ++q) t.add(__ldcg(partial + uint64_t(q) * a.part_stride + x));
  }
  if (x < NV) sh.tot[x] = t.value();
  __syncthreads();
  const float* G = sh.tot + 1 + 2 * K;
  const float* H = sh.tot + 1 + 3 * K;
  // d/d lr_k = -G_k + N exp(lr_k) L_k / Z   (N = sum_k G_k = number of sites)
  if (x < K) {
    float n = 0.f;
#pragma unroll 1
    for (uint32_t k = 0; k < K; ++k) n += G[k];
    sh.grad[x] = -G[x] + n * c.e[x] * c.ew[x] / c.z;
  }
  if (x == 32) {
    // d/d rho = -(1 - sigma) sum_k (A_k - B_k v_k / (1 - v_k))
    float acc = 0.f;
#pragma unroll 1
    for (uint32_t k = 0; k < K; ++k) acc += sh.tot[1 + k] - sh.tot[1 + K + k] * c.v[k] / (1.f - c.v[k]);
    sh.grad[K + K * J] = -(1.f - c.sig) * acc;
  }
  // d/d theta_kj = -w_kj (sum_i gamma_ik S_j(c_i) / M_k(c_i) - G_k) = -w_kj (H_kj - G_k)
  if (x >= 64 && x < 64 + K * J) sh.grad[K + x - 64] = -c.row[3 * K + x - 64] * (H[x - 64] - G[(x - 64) / J]);
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

// The forms of k_calib: an evaluation with a chunk per CTA (whose threads'
// places are their numbers: with a run-time rule, whose values spill, 512 x 1e5
// sites took 155 us)
// or by warps, and Adam steps
enum CalibForm { CHUNKS_FORM, WARPS_FORM, STEPS_FORM };

// one evaluation's results (and Adam step), by one CTA per replicate
template <uint32_t K, uint32_t J>
__device__ __forceinline__ void calib_epilogue(CalibEpilogue& sh, const CalibRow<K, J>& c, const CalibArgs& a,
                                               float* __restrict__ params, uint32_t r, float* __restrict__ nll_out,
                                               float* __restrict__ grad_out, const AdamArgs& adam) {
  constexpr uint32_t P = K + K * J + 1;
  calib_gradient<K, J>(sh, c, a, r, a.partial);
  if (threadIdx.x == 0 && nll_out) nll_out[r] = sh.tot[0];
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

// STEPS_FORM: a.steps Adam steps in a cooperative launch (an instance of its own: in
// the others the step's state would spill).  Every CTA of a replicate keeps the
// parameters and moments and makes each step itself, from the same sums in the
// same order, so a step has one wait (the sums) where parameters
// published by one CTA need a second: 0.4 ms of 200 steps over 64 x 5e4 sites.
// The sums alternate between two halves of a.partial: a CTA is at
// most one step ahead of the others.
template <uint32_t K, uint32_t J, CalibForm FORM>
__global__ void __launch_bounds__(CAL_THREADS, calib_ctas(K, J, FORM == STEPS_FORM)) k_calib(CalibArgs a, float* __restrict__ params,
                                                                               float* __restrict__ nll_out,
                                                                               float* __restrict__ grad_out,
                                                                               AdamArgs adam) {
  constexpr bool STEPS = FORM == STEPS_FORM;
  const bool by_warps = STEPS ? a.by_warps != 0u : FORM == WARPS_FORM;
  constexpr uint32_t JP = J > 4 ? 8 : 4;
  constexpr uint32_t NV = 1 + 3 * K + K * J;   // nll, A, B, G, H
  // The signature rows and the mixtures M_k(c) by class, eight copies of each
  // 16 bytes: a lane reads the copy in its own banks, so the gather is free of
  // conflicts (one copy: 2.9 lanes a bank).
  constexpr uint32_t KP = K > 4 ? 8 : 4;
  __shared__ float4 s_sig[JP / 4][CAL_MAXC * 8], s_mix[KP / 4][CAL_MAXC * 8];
  __shared__ CalibRow<K, J> s_c;
  __shared__ union { float red[CAL_WARPS][NV]; CalibEpilogue epi; } s_u;
  __shared__ uint32_t s_go;
  // what is needed after the sites (in registers it would be spilled around
  // them): the replicate, its CTAs, whether this is the first, the sums' rows
  constexpr uint32_t NO_ROW = 0xffffffffu;
  __shared__ struct { uint32_t r, parts, first, row[CAL_WARPS]; } s_at;
  // STEPS: the moments of the parameters, the step's bias corrections
  __shared__ float s_adam[2][STEPS ? K + K * J + 1 : 1];
  __shared__ AdamBias s_bias;
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t seg = a.seg0 + blockIdx.x, rep = a.seg_rep[seg];
  // this thread's chunk of the replicate and its place in it
  const uint32_t part = seg - a.rep_first_seg[rep], parts = a.rep_first_seg[rep + 1] - a.rep_first_seg[rep];
  const uint32_t unit = by_warps ? warp * parts + part : part * CAL_WARPS + warp, chunk = unit / CAL_WARPS;
  const uint32_t place = FORM == CHUNKS_FORM ? threadIdx.x : unit % CAL_WARPS * 32 + lane;
  const uint64_t end = a.site_off[rep + 1], i0 = min(a.site_off[rep] + uint64_t(chunk) * CAL_CHUNK, end);
  const uint64_t i1 = min(i0 + CAL_CHUNK, end);
  if (lane == 0) {
    const uint32_t c0 = a.rep_first_chunk[rep];
    s_at.row[warp] = chunk >= a.rep_first_chunk[rep + 1] - c0 ? NO_ROW : by_warps ? c0 * CAL_WARPS + unit : c0 + chunk;
    if (warp == 0) { s_at.r = rep; s_at.parts = parts; s_at.first = part == 0 ? 1u : 0u; }
  }
  if (STEPS) {
    if (threadIdx.x < K + K * J + 1) s_adam[0][threadIdx.x] = s_adam[1][threadIdx.x] = 0.f;
    calib_load<K, J>(s_c, a, params, rep);
  }
  for (uint32_t step = 0;; ++step) {   // a.steps evaluations (STEPS), or one
  if (STEPS) {
    if (threadIdx.x == 128) s_bias = adam_bias(adam, step);
    calib_rows<K, J>(s_c);
  } else if (a.tab) {
    if (threadIdx.x < 3 * K + K * J) s_c.row[threadIdx.x] = reinterpret_cast<const CalibRow<K, J>*>(a.tab)[rep].row[threadIdx.x];
    __syncthreads();
  } else {
    calib_tables<K, J>(s_c, a, params, rep);
  }
  const float* s_row = s_c.row;
  // a thread makes one 16-byte piece of a class's rows and writes its copies,
  // each lane of eight another copy at a time (free of conflicts)
  constexpr uint32_t QS = JP / 4, QM = KP / 4;
  if (!(STEPS && step))
    for (uint32_t x = threadIdx.x; x < a.C * QS; x += CAL_THREADS) {
      const float4 v = __ldg(reinterpret_cast<const float4*>(a.sig_rows) + x);
#pragma unroll
      for (uint32_t i = 0; i < 8; ++i) s_sig[x % QS][x / QS * 8 + ((x / QS + i) & 7u)] = v;
    }
  for (uint32_t x = threadIdx.x; x < a.C * QM; x += CAL_THREADS) {
    const uint32_t c = x / QM, k0 = x % QM * 4;
    float sg[JP], m[4];
#pragma unroll
    for (uint32_t j = 0; j < JP; j += 4) {
      const float4 v = __ldg(reinterpret_cast<const float4*>(a.sig_rows) + c * QS + j / 4);
      sg[j] = v.x; sg[j + 1] = v.y; sg[j + 2] = v.z; sg[j + 3] = v.w;
    }
#pragma unroll
    for (uint32_t i = 0; i < 4; ++i) {
      const float* w = s_row + 3 * K + min(k0 + i, K - 1) * J;
      m[i] = w[0] * sg[0];
#pragma unroll
      for (uint32_t j = 1; j < J; ++j) m[i] = __fmaf_rn(w[j], sg[j], m[i]);
      if (k0 + i >= K) m[i] = 0.f;
    }
#pragma unroll
    for (uint32_t i = 0; i < 8; ++i) s_mix[k0 / 4][c * 8 + ((c + i) & 7u)] = make_float4(m[0], m[1], m[2], m[3]);
  }
  __syncthreads();
  // epochs in pairs (packed f32x2 arithmetic); an odd K gets a padding
  // epoch of weight exp(-inf) = 0
  constexpr uint32_t KH = (K + 1) / 2;
  float2 cst[KH], dlv[KH], l1v[KH];
  auto at = [&](uint32_t k, uint32_t off, float pad) { return k < K ? s_row[off + k] : pad; };
  // the log-domain terms in base 2 (ex2 / lg2 directly, the NLL scaled back by ln 2)
  constexpr float LOG2E = 1.4426950408889634f, LN2 = 0.6931471805599453f;
#pragma unroll
  for (uint32_t h = 0; h < KH; ++h) {
    cst[h] = make_float2(LOG2E * at(2 * h, 0, 0.f), at(2 * h + 1, 0, -INFINITY) * LOG2E);
    // u_k = cst_k + a log v_k + (d - a) log(1 - v_k) = cst_k + a dlv_k + d l1v_k
    l1v[h] = make_float2(LOG2E * at(2 * h, 2 * K, 0.f), LOG2E * at(2 * h + 1, 2 * K, 0.f));
    dlv[h] = make_float2(LOG2E * at(2 * h, K, 0.f) - l1v[h].x, LOG2E * at(2 * h + 1, K, 0.f) - l1v[h].y);
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
    if (place < v0 - i0) site_at(i0 + place);
    if (place < i1 - v1) site_at(v1 + place);
    const int4* a4 = reinterpret_cast<const int4*>(a.alt) + v0 / 4;
    const int4* d4 = reinterpret_cast<const int4*>(a.depth) + v0 / 4;
    const int4* c4 = reinterpret_cast<const int4*>(a.cls) + v0 / 4;
    const uint32_t n4 = uint32_t((v1 - v0) / 4);
    // unrolled for the small shapes: by three with a chunk per CTA (512 x 1e5
    // sites 148 us, by two 150, not 169), by two otherwise (200 steps over 64 x
    // 5e4 sites 3.66 ms, by three 4.01, not 3.94)
    constexpr uint32_t UNROLL = K * J > 16 ? 1 : FORM == CHUNKS_FORM ? 3 : 2;
#pragma unroll UNROLL
    for (uint32_t q = place; q < n4; q += CAL_THREADS) site4(load4(a4 + q), load4(d4 + q), load4(c4 + q));
  }
  // the warp's sums: by a fixed tree
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
  float* const sums = STEPS && (step & 1u) ? a.partial + uint64_t(a.n_rows) * a.part_stride : a.partial;
  // row of the warp (by_warps) or of the chunk: nll, A_k, B_k, G_k, H_kj (j < J)
  const uint32_t out_row = s_at.row[warp];
  float* const out = sums + uint64_t(out_row) * a.part_stride;
#pragma unroll
  for (uint32_t q = 0; q < NV; q += 32) {
    constexpr uint32_t tail = NV % 32 ? NV % 32 : 32;
    const float v = q + 32 <= NV ? warp_transpose_sum<32>(acc + q, lane) : warp_transpose_sum<tail>(acc + q, lane);
    if (q + lane >= NV) continue;
    if (!by_warps) s_u.red[warp][q + lane] = v;
    else if (out_row != NO_ROW) out[q + lane] = v;
  }
  if (!by_warps) {
    __syncthreads();
    for (uint32_t x = threadIdx.x; x < NV && out_row != NO_ROW; x += CAL_THREADS) {
      Neu t;
      for (uint32_t w = 0; w < CAL_WARPS; ++w) t.add(s_u.red[w][x]);
      out[x] = t.value();
    }
  }
  if (!STEPS && a.tab) return;
  __threadfence();
  __syncthreads();
  const uint32_t r = s_at.r, n_parts = s_at.parts;
  if constexpr (!STEPS) {
    // the CTA that finishes the replicate's last segment runs the epilogue (the
    // count is left at zero for the next evaluation)
    if (threadIdx.x == 0) {
      s_go = atomicAdd(a.rep_done + r, 1u) + 1u == n_parts ? 1u : 0u;
      if (s_go) a.rep_done[r] = 0u;
      __threadfence();
    }
    __syncthreads();
    if (s_go) calib_epilogue<K, J>(s_u.epi, s_c, a, params, r, nll_out, grad_out, adam);
    return;
  } else {
    constexpr uint32_t P = K + K * J + 1;
    // All the replicate's sums of this step.  The CTAs are all resident (a
    // cooperative launch); should a wait run out all the same, the CTA leaves and
    // the replicate's others with it.  The first CTA alone writes results, so
    // they are those of all steps or, where it had to leave, NaN.
    if (threadIdx.x == 0) {
      uint32_t go = 0;
      atomicAdd(a.rep_done + r, 1u);
      for (uint32_t polls = 0; polls < a.wait_polls; ++polls) {
        go = arrived(*reinterpret_cast<volatile uint32_t*>(a.rep_done + r), CAL_COUNT0 + (step + 1) * n_parts);
        if (go || *reinterpret_cast<volatile uint32_t*>(a.rep_left + r) == 0u) break;
        __nanosleep(20);
      }
      __threadfence();
      if (!go) atomicExch(a.rep_left + r, 0u);
      s_go = go;
    }
    __syncthreads();
    const bool first = s_at.first != 0;
    if (!s_go) {
      const float nan = __int_as_float(0x7fc00000);
      if (first && threadIdx.x < P) params[uint64_t(r) * P + threadIdx.x] = nan;
      if (first && threadIdx.x == 0) {
        if (nll_out) nll_out[r] = nan;
        *a.status = 1u;
      }
      return;
    }
    calib_gradient<K, J>(s_u.epi, s_c, a, r, sums);
    const bool end = step + 1 == a.steps;
    if (threadIdx.x < P) {
      const float p = s_c.p[threadIdx.x] - adam_update(adam, s_bias, s_u.epi.grad[threadIdx.x], s_adam[0][threadIdx.x],
                                                       s_adam[1][threadIdx.x]);
      s_c.p[threadIdx.x] = p;
      if (end && first) params[uint64_t(r) * P + threadIdx.x] = p;
    }
    if (end) {
      if (first && threadIdx.x == 0 && nll_out) nll_out[r] = s_u.epi.tot[0];
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
  constexpr uint32_t N = sizeof(CalibRow<K, J>) / 4;
  for (uint32_t x = threadIdx.x; x < N; x += CAL_THREADS) a.tab[uint64_t(r) * N + x] = reinterpret_cast<const float*>(&s_c)[x];
}
template <uint32_t K, uint32_t J>
__global__ void __launch_bounds__(CAL_THREADS) k_calib_epilogue(CalibArgs a, float* __restrict__ params,
                                                                float* __restrict__ nll_out,
                                                                float* __restrict__ grad_out, AdamArgs adam) {
  __shared__ CalibRow<K, J> s_c;
  __shared__ CalibEpilogue s_epi;
  const uint32_t r = a.rep0 + blockIdx.x;
  constexpr uint32_t N = sizeof(CalibRow<K, J>) / 4;
  for (uint32_t x = threadIdx.x; x < N; x += CAL_THREADS)
    reinterpret_cast<float*>(&s_c)[x] = a.tab[uint64_t(r) * N + x];
  __syncthreads();
  calib_epilogue<K, J>(s_epi, s_c, a, params, r, nll_out, grad_out, adam);
}

template <uint32_t K, uint32_t J>
static void calib_run(const CalibArgs& a, uint32_t n_segs, uint32_t n_rep, float* params, float* nll, float* grad,
                      const AdamArgs& adam, cudaStream_t st) {
  static_assert(sizeof(CalibRow<K, J>) == 4 * calib_row_floats(K, J), "a row of a.tab");
  if (a.tab) k_calib_tables<K, J><<<n_rep, CAL_THREADS, 0, st>>>(a, params);
  if (a.steps == 1) {
    if (a.by_warps) k_calib<K, J, WARPS_FORM><<<n_segs, CAL_THREADS, 0, st>>>(a, params, nll, grad, adam);
    else k_calib<K, J, CHUNKS_FORM><<<n_segs, CAL_THREADS, 0, st>>>(a, params, nll, grad, adam);
  } else {
    CalibArgs aa = a;
    AdamArgs ad = adam;
    void* args[] = {&aa, &params, &nll, &grad, &ad};
    cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(k_calib<K, J, STEPS_FORM>), dim3(n_segs), dim3(CAL_THREADS), args, 0, st);
  }
  if (a.tab) k_calib_epilogue<K, J><<<n_rep, CAL_THREADS, 0, st>>>(a, params, nll, grad, adam);
  note_launch(a.tab ? 3 : 1);
}

template <uint32_t K, uint32_t J>
static int calib_resident() {
  int least = 64;
  for (const void* f : {reinterpret_cast<const void*>(k_calib<K, J, CHUNKS_FORM>), reinterpret_cast<const void*>(k_calib<K, J, WARPS_FORM>),
                        reinterpret_cast<const void*>(k_calib<K, J, STEPS_FORM>)}) {
    int n = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, f, CAL_THREADS, 0) != cudaSuccess) return 1;
    least = n < least ? n : least;
  }
  return least > 0 ? least : 1;
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
