// The FP32 samplers of pg_fast.cuh against the FP64 ones of pg_rng.cuh on the
// same Philox words: prints, per range of parameters, the draws, those the FP32
// sampler leaves undecided, and those it decides otherwise.
#include <cstdio>

#include "pg_fast.cuh"

using namespace pg;
namespace pg { void note_launch(uint32_t) {} }

struct Tally { unsigned long long draws, undecided, wrong; };

__device__ double rnd(uint32_t& s) {
  s = s * 1664525u + 1013904223u;
  uint32_t x = s ^ (s >> 15);
  x *= 0x2c1b3c6du;
  x ^= x >> 12;
  return (x + 0.5) * 0x1p-32;
}
__device__ double log_uniform(uint32_t& s, double lo, double hi) { return exp2(log2(lo) + rnd(s) * (log2(hi) - log2(lo))); }
__device__ void add(Tally* t, Tally mine) {
  atomicAdd(&t->draws, mine.draws); atomicAdd(&t->undecided, mine.undecided); atomicAdd(&t->wrong, mine.wrong);
}

enum { HALVES, RATIOS, MEANS, MASSES };

// n in [n0, n1).  HALVES: p one half or nearly (the tile tree); RATIOS: any
// quotient of two counts; MEANS: n min(p, 1 - p) in [m0, m1); MASSES: quotients
// of sums of doubles, also close to one half
__global__ void binomials(Tally* t, uint32_t seed, int mode, double n0, double n1, double m0, double m1, int per) {
  const uint32_t id = blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t s = id * 2654435761u + seed;
  Tally mine{0, 0, 0};
  for (int i = 0; i < per; ++i) {
    const uint32_t n = uint32_t(fmin(log_uniform(s, n0, n1), 4294967295.0));
    double p;
    bool flip;
    F2 pp;
    if (mode == MASSES) {
      const double y = 1e4 * (1.0 + rnd(s)) * 1.37, near = rnd(s) < 0.5 ? 1e-11 : 1.0;
      const double x = y * 0.5 * (1.0 + (rnd(s) - 0.5) * near);
      flip = x + x > y;
      p = x / y;
      int ex, ey;
      const F2 fx = f2_mantissa(flip ? y - x : x, ex), fy = f2_mantissa(y, ey);
      pp = f2_scale(f2_div(fx, fy), pow2f(ex - ey));
    } else {
      uint64_t y = 2 + uint64_t(log_uniform(s, 1.0, 4294967293.0)), x;
      if (mode == HALVES) {
        x = y / 2 + (rnd(s) < 0.5 ? 1 : 0);
      } else if (mode == RATIOS) {
        x = 1 + uint64_t(rnd(s) * double(y - 1));
      } else {
        const double mean = m0 + rnd(s) * (m1 - m0);
        y = uint64_t(log_uniform(s, 1e6, 4294967295.0));
        x = uint64_t(fmin(mean / n, 0.5) * double(y));
        if (rnd(s) < 0.5) x = y - x;
      }
      if (x < 1) x = 1;
      if (x >= y) x = y - 1;
      flip = x > y - x;
      p = double(x) / double(y);
      pp = f2_div(f2_u32(uint32_t(flip ? y - x : x)), f2_u32(uint32_t(y)));
    }
    const Stream st{Key{seed, id}, uint32_t(i), 7u, 9u, TAG_TILE_SPLIT, 0u};
    uint64_t k = 0;
    ++mine.draws;
    if (!binomial_fast(st, n, pp, flip, k)) { ++mine.undecided; continue; }
    Stream exact = st;
    if (binomial(exact, n, p) != k) ++mine.wrong;
  }
  add(t, mine);
}

__global__ void poissons(Tally* t, uint32_t seed, double l0, double l1, int per) {
  const uint32_t id = blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t s = id * 2654435761u + seed;
  Tally mine{0, 0, 0};
  for (int i = 0; i < per; ++i) {
    const double lambda = log_uniform(s, l0, l1);
    const Stream st{Key{seed, id}, uint32_t(i), 7u, 9u, TAG_EDGE_SNV, 0u};
    uint64_t k = 0;
    ++mine.draws;
    if (!poisson_fast(st, lambda, k)) { ++mine.undecided; continue; }
    Stream exact = st;
    if (poisson(exact, lambda) != k) ++mine.wrong;
  }
  add(t, mine);
}

int main() {
  Tally* d;
  if (cudaMalloc(&d, sizeof(Tally)) != cudaSuccess) return 2;
  const int blocks = 608, threads = 128, per = 400;
  auto report = [&](const char* name) {
    Tally h;
    if (cudaMemcpy(&h, d, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return false;
    std::printf("%s %llu %llu %llu\n", name, h.draws, h.undecided, h.wrong);
    return true;
  };
  struct B { const char* name; int mode; double n0, n1, m0, m1; };
  const B bs[] = {{"binomial_halves_small", HALVES, 1, 64, 0, 0},       {"binomial_halves", HALVES, 20, 16777216, 0, 0},
                  {"binomial_halves_large", HALVES, 16777216, 4294967296.0, 0, 0},
                  {"binomial_ratios", RATIOS, 20, 16777216, 0, 0},
                  {"binomial_ratios_large", RATIOS, 16777216, 4294967296.0, 0, 0},
                  {"binomial_inversion", MEANS, 20, 4294967296.0, 0, 9.99},
                  {"binomial_at_ten", MEANS, 20, 4294967296.0, 9.99, 10.01},
                  {"binomial_rejection", MEANS, 40, 4294967296.0, 10.01, 60},
                  {"binomial_masses", MASSES, 1, 4294967296.0, 0, 0}};
  uint32_t seed = 11;
  for (const B& b : bs) {
    cudaMemset(d, 0, sizeof(Tally));
    binomials<<<blocks, threads>>>(d, seed++, b.mode, b.n0, b.n1, b.m0, b.m1, per);
    if (!report(b.name)) return 2;
  }
  struct P { const char* name; double l0, l1; };
  const P ps[] = {{"poisson_tiny", 1e-6, 0.1}, {"poisson_inversion", 0.1, 9.99}, {"poisson_at_ten", 9.99, 10.01},
                  {"poisson_rejection", 10.01, 1e6}, {"poisson_large", 1e6, 1e9}};
  for (const P& p : ps) {
    cudaMemset(d, 0, sizeof(Tally));
    poissons<<<blocks, threads>>>(d, seed++, p.l0, p.l1, per);
    if (!report(p.name)) return 2;
  }
  return 0;
}
