// Exclusive prefix sums over rows of u32 / u64 values (short rows: one block
// per row; else three passes: block totals, scan of totals, block scan with
// carry-in).  Used for the
// per-context tile tables of the genome index, the per-edge mutation offsets
// and the per-bucket offsets of the locus sort.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "pg_kernels.h"

namespace pg {

constexpr int SCAN_BLOCK = 1024;   // elements per block (256 threads x 4)

template <typename T>
__device__ __forceinline__ T warp_incl_scan(T v) {
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    T n = __shfl_up_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) >= o) v += n;
  }
  return v;
}

// block-wide exclusive scan of 4 consecutive values per thread (256 threads);
// returns the block total.
template <typename T>
__device__ __forceinline__ T block_excl_scan4(T (&v)[4], T* smem /* >= 8 */) {
  T s0 = v[0], s1 = s0 + v[1], s2 = s1 + v[2], s3 = s2 + v[3];
  T incl = warp_incl_scan(s3);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 31) smem[warp] = incl;
  __syncthreads();
  T wbase = 0, total = 0;
#pragma unroll
  for (int w = 0; w < 8; ++w) { T x = smem[w]; if (w < warp) wbase += x; total += x; }
  __syncthreads();
  const T base = wbase + incl - s3;
  v[3] = base + s2; v[2] = base + s1; v[1] = base + s0; v[0] = base;
  return total;
}

template <typename T>
__global__ void k_scan_partials(const T* __restrict__ in, T* __restrict__ part, uint64_t n, int nblk) {
  __shared__ T sm[8];
  const int row = blockIdx.y;
  const uint64_t base = uint64_t(blockIdx.x) * SCAN_BLOCK + threadIdx.x * 4;
  const T* rin = in + uint64_t(row) * n;
  T v[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = (base + i < n) ? rin[base + i] : T(0);
  T tot = block_excl_scan4(v, sm);
  if (threadIdx.x == 0) part[uint64_t(row) * nblk + blockIdx.x] = tot;
}

// one block per row: exclusive scan of the block totals in place; writes row total
template <typename T>
__global__ void k_scan_totals(T* __restrict__ part, int nblk, T* __restrict__ row_total) {
  __shared__ T sm[8];
  __shared__ T carry;
  const int row = blockIdx.x;
  T* p = part + uint64_t(row) * nblk;
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  for (int b = 0; b < nblk; b += SCAN_BLOCK) {
    T v[4];
    const int base = b + threadIdx.x * 4;
#pragma unroll
    for (int i = 0; i < 4; ++i) v[i] = (base + i < nblk) ? p[base + i] : T(0);
    T tot = block_excl_scan4(v, sm);
    const T c = carry;
#pragma unroll
    for (int i = 0; i < 4; ++i) if (base + i < nblk) p[base + i] = v[i] + c;
    __syncthreads();
    if (threadIdx.x == 0) carry = c + tot;
    __syncthreads();
  }
  if (threadIdx.x == 0 && row_total) row_total[row] = carry;
}

template <typename T>
__global__ void k_scan_apply(const T* __restrict__ in, T* __restrict__ out, const T* __restrict__ part,
                             uint64_t n, int nblk) {
  __shared__ T sm[8];
  const int row = blockIdx.y;
  const uint64_t base = uint64_t(blockIdx.x) * SCAN_BLOCK + threadIdx.x * 4;
  const T* rin = in + uint64_t(row) * n;
  T* rout = out + uint64_t(row) * n;
  T v[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = (base + i < n) ? rin[base + i] : T(0);
  block_excl_scan4(v, sm);
  const T c = part[uint64_t(row) * nblk + blockIdx.x];
#pragma unroll
  for (int i = 0; i < 4; ++i) if (base + i < n) rout[base + i] = v[i] + c;
}

// One block per row: chunks of 4096 elements, the next chunk's loads under way
// while one is scanned.
constexpr int SCAN_ROW_THREADS = 1024;
template <typename T>
__global__ void __launch_bounds__(SCAN_ROW_THREADS) k_scan_row(const T* in, T* out, uint32_t n, T* row_total) {
  constexpr uint32_t WARPS = SCAN_ROW_THREADS / 32, CHUNK = 4 * SCAN_ROW_THREADS;
  __shared__ T sm[2][WARPS];        // two sets: one barrier per chunk
  const T* rin = in + uint64_t(blockIdx.x) * n;
  T* rout = out + uint64_t(blockIdx.x) * n;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  T next[4], carry = 0;
  auto load = [&](uint32_t b) {
#pragma unroll
    for (uint32_t i = 0; i < 4; ++i) {
      const uint32_t at = b + 4 * threadIdx.x + i;
      next[i] = at < n ? rin[at] : T(0);
    }
  };
  load(0);
  for (uint32_t b = 0, set = 0; b < n; b += CHUNK, set ^= 1u) {
    const T v0 = next[0], s1 = v0 + next[1], s2 = s1 + next[2], s3 = s2 + next[3];
    load(b + CHUNK);                 // (in may alias out: only this chunk is written below)
    const T incl = warp_incl_scan(s3);
    if (lane == 31) sm[set][warp] = incl;
    __syncthreads();
    const T w = sm[set][lane];       // as many warps as lanes
    const T wi = warp_incl_scan(w);
    const T base = carry + (warp ? __shfl_sync(0xffffffffu, wi, warp - 1) : T(0)) + incl - s3;
    carry += __shfl_sync(0xffffffffu, wi, WARPS - 1);
    const T o[4] = {base, T(base + v0), T(base + s1), T(base + s2)};
#pragma unroll
    for (uint32_t i = 0; i < 4; ++i) {
      const uint32_t at = b + 4 * threadIdx.x + i;
      if (at < n) rout[at] = o[i];
    }
  }
  if (threadIdx.x == 0 && row_total) row_total[blockIdx.x] = carry;
}
static_assert(SCAN_ROW_THREADS == 32 * 32, "a warp scans the warps' totals");

// Exclusive scan of `rows` rows of n elements each (in may alias out).
// `part` needs rows * ceil(n/SCAN_BLOCK) elements; row_total (optional) rows.
// Rows of up to SCAN_ROW_MAX elements take one launch: 4.1 us at 4096
// elements, 8.3 at 15000, 14.4 at 32768, where the three passes back to back
// take 12.3 at any of these sizes (and two more gaps between launches).
constexpr uint64_t SCAN_ROW_MAX = 16384;
template <typename T>
inline void scan_rows(const T* in, T* out, uint64_t n, int rows, T* part, T* row_total, cudaStream_t st) {
  const int nblk = int((n + SCAN_BLOCK - 1) / SCAN_BLOCK);
  if (n == 0) {
    if (row_total) cudaMemsetAsync(row_total, 0, sizeof(T) * rows, st);
    return;
  }
  if (n <= SCAN_ROW_MAX) {
    k_scan_row<T><<<rows, SCAN_ROW_THREADS, 0, st>>>(in, out, uint32_t(n), row_total);
    note_launch();
    return;
  }
  dim3 g(nblk, rows);
  k_scan_partials<T><<<g, 256, 0, st>>>(in, part, n, nblk);
  k_scan_totals<T><<<rows, 256, 0, st>>>(part, nblk, row_total);
  k_scan_apply<T><<<g, 256, 0, st>>>(in, out, part, n, nblk);
  note_launch(3);
}

inline uint64_t scan_part_elems(uint64_t n, int rows) {
  return uint64_t(rows) * ((n + SCAN_BLOCK - 1) / SCAN_BLOCK) + 1;
}

}  // namespace pg
