// Bulk sequencing simulation: read placement, error model and per-mutation
// alt/depth counting.
//
// Reference call site: simulate_seq (src/seq_simulation.cpp:517-601) ->
// RACES ReadSimulator<>::operator()(sequencer, mutations_list, chr_ids,
// coverage, normal_sample, purity, ...) (:371, :413, :423; RACES absent).
// The counts produced here are what the reference flattens into
// `<sample>.occurrences` and `<sample>.coverage` (src/seq_simulation.cpp:92-140).
//
// Model:
//   * per (sample, chromosome) the number of fragments is
//     floor(coverage * L / (read_len * mates)); fragment starts are i.i.d.
//     uniform over the L - read_len + 1 positions.  Starts are generated tile
//     by tile: a binary tree of binomial draws splits the fragment count over
//     the tiles (an exact multinomial), then each tile draws its starts.
//   * a fragment comes from a normal cell with the purity-derived probability,
//     otherwise from a uniformly chosen sampled leaf; the allele is uniform.
//   * paired reads: insert size from a CDF table (the reference's binomial
//     model, src/seq_simulation.cpp:431-451, or a discretised normal); the
//     second mate starts at min(start + insert - read_len, chr_end - read_len).
//   * a read covering a mutation locus adds 1 to its depth; it adds 1 to alt
//     when it carries the mutation (edge is an ancestor of the cell, same
//     allele) and the base is not hit by a substitution error, or when it
//     does not carry it and an error turns the reference into that alt base.
//     The error word of a (mate, locus) visit is a multiplicative hash of the
//     mate's word (from the XOR of the fragment's Philox block) and the
//     locus; an error happens when it is below err_thr, and the erroneous
//     base is one of the three others by the third of [0, err_thr) the word
//     falls in, the first third being the alt base.
//     Indels are not affected by substitution errors.
//
// Kernel layout (one CTA per (tile, sample); fragments in batches):
//   phase A  every thread generates fragments (one Philox block each); their
//            two mates go to shared memory in the order of their start
//            buckets (16 bp, counting sort);
//   phase B  a few lanes share a mutation record and visit the mates of the
//            buckets that may cover it, counting depth and alt in registers.
// Windows with more records than shared memory holds run a per-read loop on
// the global arrays instead.
//
// Bound by shared-memory wavefronts (78% of the pipe; about 90 per 32
// fragments: 35 for the counting sort, 35 for the visits, the draws' lookups)
// and instruction issue (61%, 10 warp instructions per fragment) around four
// barriers a batch, not by HBM.  At 155 Mbp, 100x paired, four samples with
// copy-number events (2.07e8 fragments) the launch takes 2.64 ms.  The form
// with evenly split candidate runs (a thread walks 17 or so candidates across
// record borders), a lineage walk and two table lookups per draw took 4.53 ms
// at 18.6 warp instructions per fragment; with the draws in absolute
// positions, an eight-way option comparison and the tile's copy-number tables
// gathered in the kernel, 2.88 ms.  Two fragments' draws interleaved per
// thread (2.72), one batch per tile in CTAs of 512 threads (3.25) were slower.
#include <type_traits>

#include "pg_common.cuh"
#include "pg_rng.cuh"
#include "pg_fast.cuh"
#include "pg_kernels.h"
#include "pg_scan.cuh"

namespace pg {

constexpr int SEQ_THREADS = 256;
constexpr uint32_t SEQ_CAP = 512;        // mutation records staged per CTA
constexpr uint32_t SEQ_MCAP = 2 * SEQ_FRAGS_PER_BATCH;   // mates per batch
constexpr uint32_t SEQ_BW = 16;          // start bucket width (bp)
constexpr uint32_t SEQ_NBK = 1024;       // start buckets per window (window <= 16 kbp)
static_assert(SEQ_NBK == 4 * SEQ_THREADS, "the bucket scan takes four buckets per thread");
static_assert(SEQ_GUIDE == 4 * SEQ_THREADS, "the insert table is staged by one 16-byte load per thread");
static_assert(SEQ_MCAP < 65536, "bucket offsets and a batch's counts are 16-bit");

__device__ __forceinline__ uint32_t lower_bound_rec(const SeqRec* __restrict__ recs, uint32_t n, uint32_t key) {
  uint32_t lo = 0, hi = n;
  while (lo < hi) { const uint32_t mid = (lo + hi) >> 1; if (recs[mid].locus < key) lo = mid + 1; else hi = mid; }
  return lo;
}

// Multinomial split of a chromosome's fragments over its n tiles: a binary
// tree over the padded range [0, 2^D) of tiles (D = ceil(log2 n)); the node
// with heap id h at depth d covers tiles [i 2^(D-d), (i+1) 2^(D-d)) and sends
// Binomial(count, w_left / w_node) fragments to its left half, w being the
// number of start positions of the covered tiles or, with copy-number
// events, their DNA mass in the sample (so that fragments are proportional
// to copy number across tiles; the rejection draw of the start makes them so
// within a tile).  Every node's draw uses Philox counter
// (h, chromosome, sample, TAG_TILE_SPLIT).
struct TileSplit {
  uint64_t S;            // start positions of the chromosome
  uint32_t T;            // tile size
  uint32_t nt;           // tiles of the chromosome
  const double* cum;     // mass before each tile (NULL: weigh start positions)
  double tot;            // mass of the chromosome
  __device__ __forceinline__ uint64_t w(uint64_t a, uint64_t b) const {   // start positions of tiles [a, b)
    const uint64_t x = a * T < S ? a * T : S, y = b * T < S ? b * T : S;
    return y - x;
  }
  __device__ __forceinline__ double c(uint64_t a) const { return a < nt ? cum[a] : tot; }
  // the left child's share of the node [lo, hi) (0 when the node has no mass)
  __device__ __forceinline__ double share(uint64_t n, uint64_t lo, uint64_t mid, uint64_t hi) const {
    if (cum == nullptr) {
      const uint64_t wt = w(lo, hi);
      if (n == 0 || wt == 0) return 0.0;
      return double(w(lo, mid)) / double(wt);
    }
    const double base = c(lo), wt = c(hi) - base;
    if (n == 0 || !(wt > 0.0)) return 0.0;
    return (c(mid) - base) / wt;
  }
  // the pairs of node h (n of them, tiles [lo, hi)) that go left
  __device__ __noinline__ uint64_t left(Key key, uint32_t h, uint32_t chr, uint32_t s, uint64_t n, uint64_t lo,
                                        uint64_t mid, uint64_t hi) const {
    const double p = share(n, lo, mid, hi);
    if (!(p > 0.0)) return 0;
    Stream st{key, h, chr, s, TAG_TILE_SPLIT, 0u};
    return binomial(st, n, p);
  }
  // left() from the FP32 sampler; false where that does not decide.  The
  // share p = x / y and whether it exceeds one half are taken from x and y:
  // the rounded quotient exceeds one half exactly when 2 x > y.
  __device__ __forceinline__ bool left_fast(Key key, uint32_t h, uint32_t chr, uint32_t s, uint32_t n, uint64_t lo,
                                            uint64_t mid, uint64_t hi, uint64_t& nl) const {
    F2 pp;
    bool flip;
    nl = 0;
    if (n == 0) return true;
    if (cum == nullptr) {
      const uint32_t y = uint32_t(w(lo, hi)), x = uint32_t(w(lo, mid));
      if (x == 0) return true;
      if (x >= y) { nl = n; return true; }
      flip = x > y - x;
      pp = f2_div(f2_u32(flip ? y - x : x), f2_u32(y));
    } else {
      const double base = c(lo), y = c(hi) - base, x = c(mid) - base;
      if (!(y > 0.0) || !(x > 0.0)) return true;
      if (!(x < y)) { nl = n; return true; }
      flip = x + x > y;
      int ex, ey;
      const F2 fx = f2_mantissa(flip ? y - x : x, ex), fy = f2_mantissa(y, ey);
      if (ey - ex > 60) return false;
      pp = f2_scale(f2_div(fx, fy), pow2f(ex - ey));
    }
    return binomial_fast(Stream{key, h, chr, s, TAG_TILE_SPLIT, 0u}, n, pp, flip, nl);
  }
};

// One warp per (sample, block of 64 tiles).  It walks from the root of the
// chromosome's tree to the block's node, every lane drawing the same nodes,
// then draws the block's subtree level by level with one lane per node.  The
// draws are a serial chain of at most D steps of about 2.5 us, most of them
// the same in every warp of a chromosome, which costs less than a launch per
// level: 180 us became 15 for 3 x 1 Mbp (7 levels), and at full scale
// (16 levels, 4 samples) 1.64 ms became 0.55.
constexpr uint32_t SPLIT_BLOCK_LOG = 6;   // 64 tiles per warp
constexpr uint32_t SPLIT_THREADS = 128;
// blocks per (sample, chromosome slot): as many as the longest needs
__host__ __device__ inline uint32_t split_blocks(const SeqChroms& c) {
  const uint32_t tiles = SPLIT_THREADS / 32 << SPLIT_BLOCK_LOG;
  return (c.max_tiles + tiles - 1) / tiles;
}
__device__ __forceinline__ void tile_counts_warp(const TileSplit& sp, uint32_t s, uint32_t b, uint32_t D, uint32_t chr,
                                                 uint64_t n_pairs, Key key, uint32_t* __restrict__ cnt) {
  constexpr uint32_t FULL = 0xffffffffu;
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t Db = D < SPLIT_BLOCK_LOG ? D : SPLIT_BLOCK_LOG;   // depth of the block's subtree
  if (D == 0) {   // one tile: it takes every pair
    if (lane == 0) cnt[0] = uint32_t(n_pairs);
    return;
  }
  auto draw = [&](uint32_t h, uint32_t n, uint64_t lo, uint64_t size) {
    uint64_t nl;
    if (!sp.left_fast(key, h, chr, s, n, lo, lo + (size >> 1), lo + size, nl))
      nl = sp.left(key, h, chr, s, n, lo, lo + (size >> 1), lo + size);
    return uint32_t(nl);
  };
  // root -> block node
  uint32_t n = uint32_t(n_pairs), h = 1;
  uint64_t lo = 0, size = uint64_t(1) << D;
  for (uint32_t d = Db; d < D; ++d) {
    const uint32_t nl = draw(h, n, lo, size);
    size >>= 1;
    const bool right = (uint64_t(b) << Db) >= lo + size;   // the block lies in the right half
    if (right) { n -= nl; lo += size; h = 2 * h + 1; } else { n = nl; h = 2 * h; }
  }
  // the block's subtree: lane i holds node i of the level
  for (uint32_t level = 0; level < Db; ++level, size >>= 1) {
    const uint64_t at = lo + uint64_t(lane) * size;
    uint32_t nl = 0;
    if (lane < (1u << level) && at < sp.nt) nl = draw((h << level) + lane, n, at, size);
    if (level + 1 < Db) {
      const uint32_t a = __shfl_sync(FULL, nl, lane >> 1), t = __shfl_sync(FULL, n, lane >> 1);
      n = (lane & 1u) ? t - a : a;
    } else if (lane < (1u << level)) {   // the children are tiles at and at + 1
      if (at < sp.nt) cnt[at] = nl;
      if (at + 1 < sp.nt) cnt[at + 1] = n - nl;
    }
  }
}

// block x of row `row` of the tile split (a row: a sample's chromosome slot):
// 64 tiles per warp
__device__ __forceinline__ void split_block(const SeqChroms& c, uint64_t row, uint32_t x,
                                            const double* __restrict__ mass_cum, const double* __restrict__ mass_tot,
                                            Key key, uint32_t* __restrict__ pair_cnt) {
  const uint32_t s = uint32_t(row / c.n_slots), slot = uint32_t(row % c.n_slots);
  const uint32_t b = (x * SPLIT_THREADS + threadIdx.x) >> 5;
  const uint32_t nt = c.ntiles[slot], first = c.first[slot];
  if (uint64_t(b) << SPLIT_BLOCK_LOG >= nt) return;   // whole warps
  const TileSplit sp{c.nstarts[slot], c.T, nt, mass_cum ? mass_cum + uint64_t(s) * c.n_tiles + first : nullptr,
                     mass_cum ? mass_tot[uint64_t(s) * c.n_slots + slot] : 0.0};
  tile_counts_warp(sp, s, b, c.depth[slot], c.id[slot], c.pairs[slot], key,
                   pair_cnt + uint64_t(s) * c.n_tiles + first);
}

__global__ void __launch_bounds__(SPLIT_THREADS) k_tile_split(SeqChroms c, uint64_t row0,
                                                              const double* __restrict__ mass_cum,
                                                              const double* __restrict__ mass_tot, Key key,
                                                              uint32_t* __restrict__ pair_cnt) {
  const uint32_t per = split_blocks(c);
  split_block(c, row0 + blockIdx.x / per, blockIdx.x % per, mass_cum, mass_tot, key, pair_cnt);
}

// The steps before the read kernel that wait for nothing, each a range of
// blocks: the tile split (a chain of dependent draws, so first), the tiles
// with their windows' records (two binary searches over the loci, in step),
// the records (a gather, bound by memory).  Of 3 Mbp: 16 us, against 29 as
// four launches one after the other.
template <bool SPLIT>
__global__ void __launch_bounds__(SPLIT_THREADS) k_seq_prepare(SeqChroms c, SeqTiles tiles, PlaceOut s, uint32_t n_recs,
                                                               const uint32_t* __restrict__ edge_tin,
                                                               const uint32_t* __restrict__ edge_tout, uint32_t span,
                                                               SeqRec* __restrict__ recs, uint32_t split_end,
                                                               uint32_t tiles_end, Key key,
                                                               uint32_t* __restrict__ pair_cnt) {
  if (SPLIT && blockIdx.x < split_end) {
    const uint32_t per = split_blocks(c);
    split_block(c, blockIdx.x / per, blockIdx.x % per, nullptr, nullptr, key, pair_cnt);
  } else if (blockIdx.x < tiles_end) {
    const uint32_t t = (blockIdx.x - split_end) * SPLIT_THREADS + threadIdx.x;
    if (t >= c.n_tiles) return;
    uint32_t lo = 0, hi = c.n_slots;          // last slot whose first tile is <= t
    while (hi - lo > 1) { const uint32_t mid = (lo + hi) >> 1; if (c.first[mid] <= t) lo = mid; else hi = mid; }
    const uint32_t k = t - c.first[lo], start = c.start[lo] + k * c.T, len = min(c.T, c.nstarts[lo] - k * c.T);
    tiles.start[t] = start;
    tiles.len[t] = len;
    tiles.chr_end[t] = c.end[lo];
    // records [r0, r1) of the window [start, start + len - 1 + span)
    const uint32_t end = start + len - 1 + span;
    uint32_t r0 = 0, n0 = n_recs, r1 = 0, n1 = n_recs;
    while (r0 < n0 || r1 < n1) {
      const uint32_t m0 = (r0 + n0) >> 1, m1 = (r1 + n1) >> 1;
      const uint32_t l0 = r0 < n0 ? s.locus[m0] : 0u, l1 = r1 < n1 ? s.locus[m1] : 0u;
      if (r0 < n0) { if (l0 < start) r0 = m0 + 1; else n0 = m0; }
      if (r1 < n1) { if (l1 < end) r1 = m1 + 1; else n1 = m1; }
    }
    tiles.rec_lo[t] = r0;
    tiles.rec_hi[t] = r1;
  } else {
    const uint32_t i = (blockIdx.x - tiles_end) * SPLIT_THREADS + threadIdx.x;
    if (i >= n_recs) return;
    const uint32_t e = s.edge[i];
    SeqRec r;
    r.locus = s.locus[i];
    r.tin = edge_tin[e];
    r.tout = edge_tout[e];
    r.info = uint32_t(s.allele[i]) | ((uint32_t(s.seq[i]) & 0x7fffu) << 16) | (uint32_t(s.kind[i]) << 31);
    recs[i] = r;
  }
}

// Error words.  A mate's word: the fragment's error word for mate 0, an
// odd affine map of it for mate 1.  The visit of a mate (word wm) to locus:
// a multiplicative hash (uniform, as wm is), compared with err_thr for the
// substitution error and with its thirds err_t1, err_t2 for the erroneous
// base.
__device__ __forceinline__ uint32_t mate_word(uint32_t w, uint32_t mate) {
  return mate ? w * 0x85EBCA6Bu + 0x27D4EB2Fu : w;
}
constexpr uint32_t ERR_LOCUS = 0x9E3779B1u;
__device__ __forceinline__ uint32_t err_word_at(uint32_t wm, uint32_t lc) { return (wm ^ lc) * 0xC2B2AE35u; }
__device__ __forceinline__ uint32_t err_word(uint32_t wm, uint32_t locus) { return err_word_at(wm, locus * ERR_LOCUS); }
// which of the three other bases an error word below err_thr picks
__device__ __forceinline__ uint32_t err_third(const SeqParams& prm, uint32_t e) {
  return e < prm.err_t1 ? 0u : (e < prm.err_t2 ? 1u : 2u);
}

// does allele instance y of the read's cell carry the mutation placed on
// instance x with order key key_m (tin of its edge << 16 | order on the edge)?
// y carries it when y is x, or when y descends from x through copies made
// after the mutation (a copy's key exceeds the mutation's: both lie on the
// cell's root path, where tin grows with depth)
__device__ __forceinline__ bool inst_carries(const SeqParams& prm, uint32_t y, uint32_t x, uint64_t key_m) {
  if (y == x) return true;
  if (!prm.has_cna) return false;
  for (uint32_t q = __ldg(prm.chain_off + y), e = __ldg(prm.chain_off + y + 1); q < e; ++q)
    if (__ldg(prm.chain_anc + q) == x) return __ldg(prm.chain_key + q) > key_m;
  return false;
}

// did the visit of a mate (word wm) observe the alt base?
__device__ __forceinline__ bool observed(const SeqParams& prm, uint32_t tin, uint32_t tout, uint32_t info,
                                         uint32_t cell, uint32_t inst, uint32_t wm, uint32_t locus) {
  // the cell is in the edge's subtree when tin <= cell < tout (one unsigned compare)
  // branch-free but for the lineage walk of a copied instance: the error
  // word is computed for indels too, and the caller evaluates every
  // candidate mate (covering or not), so that a warp does not diverge.
  // A copy has a larger instance number than its source, and instances 0
  // and 1 have no source: the walk is needed only when inst > max(x, 1).
  const bool sub = cell - tin < tout - tin;
  const uint32_t x = info & 0xffffu;
  bool carried = sub && inst == x;
  if (sub && inst > max(x, 1u) && prm.has_cna)
    carried = inst_carries(prm, inst, x, (uint64_t(tin) << 16) | ((info >> 16) & 0x7fffu));
  const uint32_t e = err_word(wm, locus);
  const bool snv = carried ? e >= prm.err_thr : e < prm.err_t1;
  return (info >> 31) ? carried : snv;
}

// One fragment's draws: mate starts, source cell, allele instance and its
// error word, all from ONE Philox4x32-10 block r (counter (j, t, s, TAG_PAIR)):
//   r.x  the start: uniform in the tile; with copy-number events, when the
//        tile meets several atoms, the part by its mass (31-bit thresholds)
//        and the start uniform in the part from the word's residual within
//        the part's threshold interval (exact integer arithmetic)
//   r.y  the cell: normal when below normal_thr, else a sampled leaf; with
//        copy-number events the cell option (normal cells or a leaf class)
//        by its copies in the part's atom
//   r.z  the insert size (31-bit thresholds of its CDF)
//   r.w  the allele instance, uniform among the n covering ones
//        (floor(r.w n / 2^32)), then the leaf, uniform in its class, from the
//        fraction that draw leaves (the low word of r.w n): the two indices
//        use disjoint information of the word
//   r.x ^ r.y ^ r.z ^ r.w  the fragment's error word
// Without copy-number events the instance is allele 0 or 1 and the leaf is
// uniform over the sample's leaves.
struct Fragment {
  uint32_t p0, p1, cell, inst, w;
};

// The copy-number draw tables of one (tile, sample) staged in shared memory:
// the tile's parts with their thresholds and, per part, a CnRow's tables for
// its atom, the local ids numbered through over the parts.  With them a
// fragment's instance draw needs no lookup and a record can hold the set of
// instances that carry it as a bit mask over the ids.  Almost every tile lies
// in one atom: its tables come as a row made once per call, one load after
// the tile's header, where reading them here through part, atom and class
// held the CTA back for five dependent loads.
constexpr uint32_t SEQ_CN_PARTS = 4;
struct CnCache {
  uint4 othr[SEQ_CN_PARTS][SEQ_CN_OPTS];       // option thresholds (.x; the stride of opt, so that one offset serves both)
  uint4 opt[SEQ_CN_PARTS][SEQ_CN_OPTS];        // covering instances, leaves, first leaf, tag of the first instance
  uint4 linst[SEQ_CN_IDS / 4];
  uint32_t pstart[SEQ_CN_PARTS], plen[SEQ_CN_PARTS], pthr[SEQ_CN_PARTS];
  uint32_t n_parts, n_ids;
};

// one option's draw table entries in an atom: its threshold, {covering
// instances, leaves, first leaf, 0} and the offset of its instance list
__device__ __forceinline__ uint32_t cn_option(const SeqParams& prm, const SeqSample& sm, uint32_t atom, uint32_t o,
                                              uint4& op, uint32_t& ioff) {
  const uint32_t ai = atom * prm.n_classes + prm.opt_class[sm.opt_off + o];
  ioff = prm.atom_ioff[ai];
  op = make_uint4(prm.atom_icnt[ai], prm.opt_nleaf[sm.opt_off + o], prm.opt_leaf_off[sm.opt_off + o], 0u);
  return o + 1 < sm.n_opt ? prm.opt_cdf[sm.opt_cdf_off + atom * sm.n_opt + o] : 0xffffffffu;
}
// the mate tag of local id l (see ReadSmem), or that of a dropped fragment
__device__ __forceinline__ uint32_t cn_tag(uint32_t icnt, uint32_t l) { return icnt ? 0x10000u << (l & 15u) : 0x8000u; }

// one warp fills the cache of a tile of up to SEQ_CN_PARTS parts (and the
// sample of up to SEQ_CN_OPTS options); linst is incomplete when n_ids
// exceeds SEQ_CN_IDS
__device__ __forceinline__ void fill_cn_cache(CnCache& c, const SeqParams& prm, const SeqSample& sm, uint32_t t,
                                              uint32_t s, uint32_t lane) {
  const uint32_t pb = prm.part_off[t], pn = prm.part_off[t + 1] - pb;
  if (lane < pn) {
    c.pstart[lane] = prm.part_start[pb + lane];
    c.plen[lane] = prm.part_len[pb + lane];
    c.pthr[lane] = prm.part_cdf[uint64_t(s) * prm.n_parts + pb + lane];
  }
  const uint32_t p = lane / SEQ_CN_OPTS, o = lane % SEQ_CN_OPTS;   // SEQ_CN_PARTS x SEQ_CN_OPTS = 32 lanes
  uint32_t thr = 0xffffffffu, ioff = 0;
  uint4 op = make_uint4(0u, 0u, 0u, 0u);
  if (p < pn && o < sm.n_opt) thr = cn_option(prm, sm, prm.part_atom[pb + p], o, op, ioff);
  const uint32_t incl = warp_incl_scan(op.x), id0 = incl - op.x;
  op.w = cn_tag(op.x, id0);
  c.othr[p][o].x = thr;
  c.opt[p][o] = op;
  uint32_t* linst = reinterpret_cast<uint32_t*>(c.linst);
  for (uint32_t i = 0; i < op.x && id0 + i < SEQ_CN_IDS; ++i) linst[id0 + i] = prm.gc.inst_list[ioff + i];
  if (lane == 31) { c.n_parts = pn; c.n_ids = incl; }
}
static_assert(SEQ_CN_PARTS * SEQ_CN_OPTS == 32 && SEQ_CN_OPTS == 8, "one lane per (part, option)");

// the same tables of whole atoms: eight lanes per (sample, atom)
__global__ void k_cn_rows(SeqParams prm, const SeqSample* __restrict__ samples, uint32_t n_samples,
                          CnRow* __restrict__ rows) {
  const uint64_t row = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) / SEQ_CN_OPTS;
  const uint32_t o = threadIdx.x % SEQ_CN_OPTS;
  const bool mine = row < uint64_t(n_samples) * prm.n_atoms;
  const SeqSample sm = samples[mine ? row / prm.n_atoms : 0];
  const bool fits = sm.n_opt <= SEQ_CN_OPTS;
  uint32_t thr = 0xffffffffu, ioff = 0;
  uint4 op = make_uint4(0u, 0u, 0u, 0u);
  if (mine && fits && o < sm.n_opt) thr = cn_option(prm, sm, uint32_t(row % prm.n_atoms), o, op, ioff);
  uint32_t incl = op.x;
#pragma unroll
  for (uint32_t d = 1; d < SEQ_CN_OPTS; d <<= 1) {
    const uint32_t v = __shfl_up_sync(0xffffffffu, incl, d, SEQ_CN_OPTS);
    if (o >= d) incl += v;
  }
  if (!mine) return;
  const uint32_t id0 = incl - op.x;
  op.w = cn_tag(op.x, id0);
  CnRow& r = rows[row];
  r.thr[o] = thr;
  r.opt[o] = op;
  for (uint32_t i = 0; i < op.x && id0 + i < SEQ_CN_IDS; ++i) r.linst[id0 + i] = prm.gc.inst_list[ioff + i];
  if (o == SEQ_CN_OPTS - 1) r.n_ids = fits ? incl : 0xffffffffu;
}

// cdf_lookup for tables of at most NMAX (a power of two) thresholds: the
// count of thresholds <= u >> 1 by binary lifting, without a data-dependent
// loop (the same index as cdf_lookup for sorted thresholds)
template <uint32_t NMAX>
__device__ __forceinline__ uint32_t cdf_lookup_small(const uint32_t* thr, uint32_t n, uint32_t u) {
  const uint32_t v = u >> 1;
  uint32_t lo = 0;
#pragma unroll
  for (uint32_t step = NMAX; step >= 1; step >>= 1)
    if (lo + step <= n && thr[lo + step - 1] <= v) lo += step;
  return lo < n ? lo : n - 1;
}

// start offset in a part of length plen from the word u that selected the
// part, whose 31-bit value lies in the part's threshold interval [lo, hi)
__device__ __forceinline__ uint32_t part_offset(uint32_t u, uint32_t lo, uint32_t hi, uint32_t plen) {
  return uint32_t((uint64_t((u >> 1) - lo) * plen) / uint64_t(hi - lo));
}

// (KeyT: Key, or the precomputed RoundKeys of the same key)
__device__ __forceinline__ U4 pair_block(const Key& key, uint32_t j, uint32_t t, uint32_t s) {
  return philox(key.k0, key.k1, j, t, s, TAG_PAIR);
}
__device__ __forceinline__ U4 pair_block(const RoundKeys& rk, uint32_t j, uint32_t t, uint32_t s) {
  return philox(rk, j, t, s, TAG_PAIR);
}

// index of the insert size: by the guide (one lookup, but where several
// thresholds share the word's cell) or by binary search
template <bool GUIDE>
__device__ __forceinline__ uint32_t insert_index(const SeqParams& prm, const uint32_t* guide, uint32_t u) {
  if (!GUIDE) return cdf_lookup(prm.ins_cdf, prm.n_ins, u);
  const uint32_t g = guide[u >> 22];
  const bool past = (u << 10) > (g | 0x7ffu);
  uint32_t k = (g & 1023u) + (past ? 1u : 0u);
  if (past && (g & 1024u))
    while (__ldg(prm.ins_cdf + k) <= (u >> 1)) ++k;   // the last threshold is 2^31, past every word
  return k;
}

// CN: with copy-number events (0, 1), or as prm.has_cna says (-1)
template <bool GUIDE, int CN = -1, class KeyT>
__device__ __forceinline__ Fragment make_fragment(const KeyT& key, uint32_t j, uint32_t t, uint32_t s, uint32_t start,
                                                  uint32_t len, uint32_t ce, const SeqSample& sm,
                                                  const uint32_t* __restrict__ leaf_tin, const SeqParams& prm,
                                                  const uint32_t* guide) {
  const U4 r = pair_block(key, j, t, s);
  Fragment f;
  const uint32_t R = prm.read_len;
  if (CN == 0 || (CN < 0 && !prm.has_cna)) {
    f.p0 = start + __umulhi(r.x, len);
    const bool normal = sm.all_normal || r.y < sm.normal_thr;
    f.inst = __umulhi(r.w, prm.n_alleles);
    f.cell = normal ? prm.normal_tin
                    : __ldg(leaf_tin + sm.leaf_off + __umulhi(r.w * prm.n_alleles, sm.n_leaves));
  } else {
    const uint32_t pb = __ldg(prm.part_off + t), pn = __ldg(prm.part_off + t + 1) - pb;
    uint32_t part = pb;
    if (pn > 1) {
      const uint32_t* thr = prm.part_cdf + uint64_t(s) * prm.n_parts + pb;
      const uint32_t k = cdf_lookup(thr, pn, r.x);
      part = pb + k;
      f.p0 = __ldg(prm.part_start + part) +
             part_offset(r.x, k ? __ldg(thr + k - 1) : 0u, __ldg(thr + k), __ldg(prm.part_len + part));
    } else {
      f.p0 = __ldg(prm.part_start + part) + __umulhi(r.x, __ldg(prm.part_len + part));
    }
    const uint32_t atom = __ldg(prm.part_atom + part);
    const uint32_t o = sm.opt_off + cdf_lookup(prm.opt_cdf + sm.opt_cdf_off + atom * sm.n_opt, sm.n_opt, r.y);
    const uint32_t nl = __ldg(prm.opt_nleaf + o);
    const uint32_t ai = atom * prm.n_classes + __ldg(prm.opt_class + o);
    const uint32_t icnt = __ldg(prm.atom_icnt + ai);
    f.inst = icnt ? uint32_t(__ldg(prm.gc.inst_list + __ldg(prm.atom_ioff + ai) + __umulhi(r.w, icnt))) : 0xffffu;
    f.cell = nl ? __ldg(prm.cls_leaf_tin + __ldg(prm.opt_leaf_off + o) + __umulhi(r.w * icnt, nl)) : prm.normal_tin;
  }
  f.w = r.x ^ r.y ^ r.z ^ r.w;
  f.p1 = f.p0;
  if (prm.paired) {
    uint32_t p1 = f.p0 + prm.ins_min + insert_index<GUIDE>(prm, guide, r.z) - R;
    if (p1 > ce - R) p1 = ce - R;
    f.p1 = p1;
  }
  return f;
}

// shared memory of one read CTA
struct ReadSmem {
  // records of the window: offset in the window << 16 | kind, tin, tout - tin,
  // and the mask of the local ids that carry the record << 16 (or, where the
  // instances have no local ids, the record's info word); their first and
  // last-plus-one candidate buckets
  uint4 s_rec[SEQ_CAP];
  uint32_t s_bnd[SEQ_CAP];
  uint2 s_cnt[SEQ_CAP];          // depth, alt
  // mates of the batch in start-bucket order
  uint2 s_mcw[SEQ_MCAP];         // source cell (Euler index), the mate's error word
  uint32_t s_mpi[SEQ_MCAP];      // start offset in the window | local id's bit (or the instance) << 16 (a
                                 //   dropped fragment: offset with bit 15 set)
  uint4 s_hist[SEQ_NBK / 4];     // mates per start bucket; all zero between batches
  uint16_t s_boff[SEQ_NBK + 4];  // first mate of each bucket
  uint4 s_guide[SEQ_GUIDE / 4];
  uint32_t s_scan[SEQ_THREADS / 32];
  CnCache s_cn;
};

// One work item: the n_pairs fragments of tile t (window [start, ...),
// records [lo, lo + nw) of g_recs) for sample s, counted into the rows
// g_alt_row / g_dep_row (indexed by record).  Called by every thread of the
// CTA with the same arguments; s_hist is all zero on entry and on return.
//
// The fragments go through in batches.  Phase A draws them, a histogram's
// atomics giving each mate its rank in its 16 bp start bucket, and places the
// mates in bucket order.  Phase B takes a record per group of lanes: its candidate
// mates (those starting in the buckets of [L - R + 1, L]) are one contiguous
// run, dealt out to the record's lanes.
// Instruction issue bounds the kernel, so what a visit needs is prepared per
// record: "the mate's instance carries the mutation" is one bit of the
// record's mask, and the error thresholds of an indel are 0.
template <class KeyT>
__device__ __forceinline__ void read_tile(ReadSmem& sh, const SeqRec* __restrict__ g_recs, uint32_t t, uint32_t s,
                                          uint32_t atom, uint32_t n_pairs, uint32_t lo, uint32_t nw, uint32_t start, uint32_t len,
                                          uint32_t ce, const SeqSample& sm, const uint32_t* __restrict__ leaf_tin,
                                          const SeqParams& prm, const KeyT& key, uint32_t* __restrict__ g_alt_row,
                                          uint32_t* __restrict__ g_dep_row) {
  const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
  constexpr uint32_t WARPS = SEQ_THREADS / 32;
  if (nw == 0 || n_pairs == 0) return;       // nothing to count in this window
  const uint32_t R = prm.read_len;
  const uint32_t wlen = len - 1 + prm.span;   // the window is [start, start + wlen)
  const uint32_t nbk = (wlen + SEQ_BW - 1) / SEQ_BW;
  uint32_t* galt = g_alt_row + lo;
  uint32_t* gdep = g_dep_row + lo;
  const SeqRec* grec = g_recs + lo;
  const bool ins_smem = prm.paired && prm.n_ins <= SEQ_GUIDE_INS;

  if (nw > SEQ_CAP || nbk > SEQ_NBK || wlen >= 32768u) {
    // dense or long window: per-read loop over the global records
    for (uint32_t j = tid; j < n_pairs; j += SEQ_THREADS) {
      const Fragment f = make_fragment<false>(key, j, t, s, start, len, ce, sm, leaf_tin, prm, nullptr);
      if (f.inst == 0xffffu) continue;   // dropped: no covering instance
      for (uint32_t mate = 0; mate < (prm.paired ? 2u : 1u); ++mate) {
        const uint32_t a = mate ? f.p1 : f.p0;
        for (uint32_t i = lower_bound_rec(grec, nw, a); i < nw; ++i) {
          const SeqRec r = grec[i];
          if (r.locus >= a + R) break;
          atomicAdd(gdep + i, 1u);
          if (observed(prm, r.tin, r.tout, r.info, f.cell, f.inst, mate_word(f.w, mate), r.locus))
            atomicAdd(galt + i, 1u);
        }
      }
    }
    return;
  }

  // copy-number draws from shared memory when the tile's tables fit
  const bool row = prm.has_cna && atom != 0xffffffffu;
  const bool parts = prm.has_cna && !row && sm.n_opt <= SEQ_CN_OPTS &&
                     prm.part_off[t + 1] - prm.part_off[t] <= SEQ_CN_PARTS;
  // (the first records are on their way meanwhile)
  SeqRec r{};
  if (tid / 4 < nw) r = grec[tid / 4];
  if (row) {
    const CnRow& cr = prm.cn_rows[uint64_t(s) * prm.n_atoms + atom];
    if (tid < SEQ_CN_OPTS) sh.s_cn.othr[0][tid].x = __ldg(cr.thr + tid);
    else if (tid < 2 * SEQ_CN_OPTS) sh.s_cn.opt[0][tid - SEQ_CN_OPTS] = __ldg(cr.opt + tid - SEQ_CN_OPTS);
    else if (tid < 2 * SEQ_CN_OPTS + SEQ_CN_IDS / 4)
      sh.s_cn.linst[tid - 2 * SEQ_CN_OPTS] = __ldg(reinterpret_cast<const uint4*>(cr.linst) + tid - 2 * SEQ_CN_OPTS);
    else if (tid == 31) sh.s_cn.n_ids = __ldg(&cr.n_ids);
  } else if (parts && warp == 0) {
    fill_cn_cache(sh.s_cn, prm, sm, t, s, lane);
  }
  if (ins_smem) sh.s_guide[tid] = __ldg(reinterpret_cast<const uint4*>(prm.ins_guide) + tid);
  __syncthreads();
  const int cn = !prm.has_cna ? 0 : !((row || parts) && sh.s_cn.n_ids <= SEQ_CN_IDS) ? 2 : row ? 1 : 3;
  // the records, four threads each (they share the walk over the local ids)
  const uint32_t n_ids = cn & 1 ? sh.s_cn.n_ids : 0u;
  for (uint32_t i0 = 0; i0 < nw; i0 += SEQ_THREADS / 4) {
    const uint32_t i = i0 + tid / 4, sub = tid % 4;
    if (i0 > 0 && i < nw) r = grec[i];
    const uint32_t x = r.info & 0xffffu;
    const uint64_t km = (uint64_t(r.tin) << 16) | ((r.info >> 16) & 0x7fffu);
    uint32_t m = cn == 0 && x < SEQ_CN_IDS ? 1u << x : 0u;
    if (i < nw)
      for (uint32_t l = sub; l < n_ids; l += 4) {
        // a copy has a larger instance number than its source, and instances
        // 0 and 1 have no source
        const uint32_t y = reinterpret_cast<const uint32_t*>(sh.s_cn.linst)[l];
        if (y == x || (y > max(x, 1u) && inst_carries(prm, y, x, km))) m |= 1u << l;
      }
    m |= __shfl_xor_sync(0xffffffffu, m, 1);
    m |= __shfl_xor_sync(0xffffffffu, m, 2);
    if (i < nw && sub == 0) {
      const uint32_t off = r.locus - start;
      sh.s_rec[i] = make_uint4((off << 16) | (r.info >> 31), r.tin, r.tout - r.tin, cn == 2 ? r.info : m << 16);
      sh.s_bnd[i] = (off + 1 >= R ? off + 1 - R : 0u) / SEQ_BW | (min(off / SEQ_BW, nbk - 1) + 1) << 16;
      sh.s_cnt[i] = make_uint2(0u, 0u);
    }
  }

  // phase B's lanes per record: as many as take all records in one pass (a
  // second, nearly empty pass holds the CTA's other warps at the barrier), but
  // 2 to 16, and 4 from three passes on.  Against 4 throughout: a batch of
  // 24 genomes (5 to 60 records a window) 9.86 -> 9.38 ms, 81 records a
  // window the same within 0.3%.
  const uint32_t lsh = nw <= 16 ? 4u : nw <= 32 ? 3u : nw <= 64 ? 2u : nw <= 128 ? 1u : 2u;
  const uint32_t lanes = 1u << lsh, sub = tid & (lanes - 1u);
  constexpr uint32_t per_batch = SEQ_MCAP / 2;
  constexpr uint32_t FPT = per_batch / SEQ_THREADS;   // fragments per thread and batch
  uint32_t* hist = reinterpret_cast<uint32_t*>(sh.s_hist);
  const bool paired = prm.paired != 0;
  for (uint32_t b0 = 0; b0 < n_pairs; b0 += per_batch) {
    const uint32_t nb_pairs = min(per_batch, n_pairs - b0);
    // phase A: fragments stay in registers (mate offsets, both < 2^15, and
    // bucket ranks, both < 2^16, packed in pairs); each mate takes its rank
    // within its start bucket from the histogram's atomic.  (No barrier
    // since the last batch's phase B: what this writes, the histogram, was
    // cleared by the last scan.)
    uint32_t o01[FPT], ca[FPT], fi[FPT], fw[FPT], rk01[FPT];
    // one instance of the draw code per (copy-number path, insert table)
    // pair, chosen once per tile: the unrolled loop holds only that path.
    // The draws are make_fragment's, as window offsets and mate tags, and run
    // in the lanes past the batch's end too (only their ranks are not taken).
    auto gen = [&](auto path, auto insert) {
      constexpr int CN = decltype(path)::value;           // 0 none, 1 one atom, 3 several, 2 tables in global memory
      constexpr bool GUIDE = decltype(insert)::value;     // (paired)
      const CnCache& cc = sh.s_cn;
      const uint32_t* guide = reinterpret_cast<const uint32_t*>(sh.s_guide);
      const uint32_t last = ce - R - start, ins0 = prm.ins_min - R;
      const uint32_t t3 = CN == 1 ? cc.othr[0][3].x : 0u;
#pragma unroll
      for (uint32_t q = 0; q < FPT; ++q) {
        const uint32_t k = tid + q * SEQ_THREADS;
        if (!__any_sync(0xffffffffu, k < nb_pairs)) break;
        uint32_t o0, o1 = 0;
        if constexpr (CN == 2) {
          const Fragment f = make_fragment<GUIDE, 1>(key, b0 + k, t, s, start, len, ce, sm, leaf_tin, prm, guide);
          o0 = f.p0 - start; o1 = f.p1 - start;
          ca[q] = f.cell;
          fi[q] = f.inst == 0xffffu ? 0x8000u : f.inst << 16;
          fw[q] = f.w;
        } else {
          const U4 r = pair_block(key, b0 + k, t, s);
          uint32_t cell = prm.normal_tin;
          if constexpr (CN == 0) {
            o0 = __umulhi(r.x, len);
            fi[q] = 0x10000u << (__umulhi(r.w, prm.n_alleles) & 15u);
            if (!sm.all_normal && r.y >= sm.normal_thr)
              cell = __ldg(leaf_tin + sm.leaf_off + __umulhi(r.w * prm.n_alleles, sm.n_leaves));
          } else {
            uint32_t part = 0;
            if constexpr (CN == 1) {
              o0 = __umulhi(r.x, len);
            } else {
              part = cdf_lookup_small<SEQ_CN_PARTS>(cc.pthr, cc.n_parts, r.x);
              o0 = cc.pstart[part] - start +
                   part_offset(r.x, part ? cc.pthr[part - 1] : 0u, cc.pthr[part], cc.plen[part]);
            }
            // the option: the number of thresholds at or below the 31-bit
            // word, in units of the tables' stride
            const char* thr = reinterpret_cast<const char*>(cc.othr[part]);
            const uint32_t v = r.y >> 1;
            uint32_t o = (CN == 1 ? t3 : cc.othr[part][3].x) <= v ? 64u : 0u;
            if (*reinterpret_cast<const uint32_t*>(thr + o + 16) <= v) o += 32u;
            if (*reinterpret_cast<const uint32_t*>(thr + o) <= v) o += 16u;
            const uint4 op = *reinterpret_cast<const uint4*>(reinterpret_cast<const char*>(cc.opt[part]) + o);
            fi[q] = op.w << __umulhi(r.w, op.x);
            if (op.y) cell = __ldg(prm.cls_leaf_tin + op.z + __umulhi(r.w * op.x, op.y));
          }
          ca[q] = cell;
          fw[q] = r.x ^ r.y ^ r.z ^ r.w;
          if (GUIDE || paired) o1 = min(o0 + ins0 + insert_index<GUIDE>(prm, guide, r.z), last);
        }
        o01[q] = o0 | (o1 << 16);
        if (k < nb_pairs) {
          uint32_t rk = atomicAdd(hist + o0 / SEQ_BW, 1u);
          if (GUIDE || paired) rk |= atomicAdd(hist + o1 / SEQ_BW, 1u) << 16;
          rk01[q] = rk;
        }
      }
    };
    using T0 = std::integral_constant<int, 0>;
    using T1 = std::integral_constant<int, 1>;
    using T2 = std::integral_constant<int, 2>;
    using T3 = std::integral_constant<int, 3>;
    using YES = std::true_type;
    using NO = std::false_type;
    if (cn == 0) { if (ins_smem) gen(T0{}, YES{}); else gen(T0{}, NO{}); }
    else if (cn == 1) { if (ins_smem) gen(T1{}, YES{}); else gen(T1{}, NO{}); }
    else if (cn == 2) { if (ins_smem) gen(T2{}, YES{}); else gen(T2{}, NO{}); }
    else { if (ins_smem) gen(T3{}, YES{}); else gen(T3{}, NO{}); }
    __syncthreads();
    // bucket offsets: exclusive scan of the 1024 counts, four per thread,
    // the counts cleared for the next batch
    {
      const uint4 c = sh.s_hist[tid];
      sh.s_hist[tid] = make_uint4(0u, 0u, 0u, 0u);
      const uint32_t c1 = c.x + c.y, c2 = c1 + c.z, c3 = c2 + c.w;
      const uint32_t incl = warp_incl_scan(c3);
      if (lane == 31) sh.s_scan[warp] = incl;
      __syncthreads();
      uint32_t base = incl - c3;
#pragma unroll
      for (uint32_t w = 0; w < WARPS - 1; ++w) base += w < warp ? sh.s_scan[w] : 0u;
      const uint32_t a0 = base, a1 = base + c.x, a2 = base + c1, a3 = base + c2;
      *reinterpret_cast<uint2*>(sh.s_boff + 4 * tid) = make_uint2(a0 | (a1 << 16), a2 | (a3 << 16));
      if (tid == SEQ_THREADS - 1) sh.s_boff[SEQ_NBK] = uint16_t(base + c3);
    }
    __syncthreads();
    // scatter the mates in start-bucket order
#pragma unroll
    for (uint32_t q = 0; q < FPT; ++q) {
      const uint32_t k = tid + q * SEQ_THREADS;
      if (k < nb_pairs) {
        const uint32_t o0 = o01[q] & 0xffffu, o1 = o01[q] >> 16;
        const uint32_t x0 = sh.s_boff[o0 / SEQ_BW] + (rk01[q] & 0xffffu);
        sh.s_mpi[x0] = o0 | fi[q]; sh.s_mcw[x0] = make_uint2(ca[q], fw[q]);
        if (paired) {
          const uint32_t x1 = sh.s_boff[o1 / SEQ_BW] + (rk01[q] >> 16);
          sh.s_mpi[x1] = o1 | fi[q]; sh.s_mcw[x1] = make_uint2(ca[q], mate_word(fw[q], 1u));
        }
      }
    }
    __syncthreads();
    // phase B: 1 << lsh lanes per record
    const uint32_t err_thr = prm.err_thr, err_t1 = prm.err_t1, R16 = R << 16, lc0 = start * ERR_LOCUS;
    auto visits = [&](auto ids_tag) {
      constexpr bool IDS = decltype(ids_tag)::value;
      for (uint32_t i0 = 0; i0 < nw; i0 += SEQ_THREADS >> lsh) {
        const uint32_t i = i0 + (tid >> lsh);
        uint32_t acc = 0;                    // depth | alt << 16 (a batch holds 2560 mates)
        if (i < nw) {
          const uint4 r = sh.s_rec[i];
          const uint32_t bnd = sh.s_bnd[i], e = sh.s_boff[bnd >> 16];
          const uint32_t off16 = r.x & 0xffff0000u, lc = (r.x >> 16) * ERR_LOCUS + lc0;
          const uint32_t thr = (r.x & 1u) ? 0u : err_thr, t1 = (r.x & 1u) ? 0u : err_t1;
#pragma unroll 2
          for (uint32_t k = sh.s_boff[bnd & 0xffffu] + sub; k < e; k += lanes) {
            const uint32_t pi = sh.s_mpi[k];
            const uint2 cw = sh.s_mcw[k];
            // the mate covers L when its start o is in (L - R, L] (unsigned: o > off wraps)
            const bool cov = off16 - pi * 0x10000u < R16;
            // the cell is in the edge's subtree when tin <= cell < tout
            bool carried = cw.x - r.y < r.z;
            if constexpr (IDS) {
              carried = carried && (pi & r.w) != 0u;   // (r.w has no bits below 16)
            } else {
              const uint32_t y = pi >> 16, x = r.w & 0xffffu;
              if (carried && y > max(x, 1u))
                carried = inst_carries(prm, y, x, (uint64_t(r.y) << 16) | ((r.w >> 16) & 0x7fffu));
              else
                carried = carried && y == x;
            }
            // carried: the alt base unless an error hits it; else an error of
            // the first third shows it (an indel has neither)
            const bool ob = (err_word_at(cw.y, lc) < (carried ? thr : t1)) != carried;
            const uint32_t one = ob ? 0x10001u : 1u;
            if (cov) acc += one;
          }
        }
        for (uint32_t o = lanes >> 1; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (acc && sub == 0) {
          uint2 c = sh.s_cnt[i];
          c.x += acc & 0xffffu;
          c.y += acc >> 16;
          sh.s_cnt[i] = c;
        }
      }
    };
    if (cn == 2) visits(NO{}); else visits(YES{});
  }
  __syncthreads();
  for (uint32_t i = tid; i < nw; i += SEQ_THREADS) {
    const uint2 c = sh.s_cnt[i];
    if (c.x) {
      atomicAdd(gdep + i, c.x);
      if (c.y) atomicAdd(galt + i, c.y);
    }
  }
}


__global__ void __launch_bounds__(SEQ_THREADS, 4) k_reads(const SeqRec* __restrict__ g_recs, SeqTiles tiles,
                                                          const uint32_t* __restrict__ pair_cnt,
                                                          const SeqSample* __restrict__ samples,
                                                          const uint32_t* __restrict__ leaf_tin, SeqParams prm,
                                                          RoundKeys key, uint64_t n_recs, uint32_t* __restrict__ g_alt,
                                                          uint32_t* __restrict__ g_dep) {
  __shared__ __align__(16) ReadSmem sh;
  const uint32_t t = blockIdx.x, s = blockIdx.y;
  sh.s_hist[threadIdx.x] = make_uint4(0u, 0u, 0u, 0u);
  const uint32_t lo = tiles.rec_lo[t];
  const SeqSample sm = samples[s];
  const uint32_t atom = prm.has_cna ? prm.tile_atom[t] : 0u;
  read_tile(sh, g_recs, t, s, atom, pair_cnt[uint64_t(s) * tiles.n_tiles + t], lo, tiles.rec_hi[t] - lo, tiles.start[t],
            tiles.len[t], tiles.chr_end[t], sm, leaf_tin, prm, key, g_alt + uint64_t(s) * n_recs,
            g_dep + uint64_t(s) * n_recs);
}

constexpr uint64_t MAX_GRID_X = 0x7fffffffu;
static inline unsigned nblk(uint64_t n, int b = 256) { return unsigned((n + b - 1) / b); }

// ------------------------------------------------------------ SAM reads
// The bases of one mate starting at reference position p: the reference with
// the carried SNVs (alt base) and indels (inserted bases; skipped deleted
// bases, anchored at the base before them), and a substitution wherever the
// visit's error word is below the threshold.  A substitution picks one of the
// three other bases by the third of [0, err_thr) its word falls in; at an SNV
// site the first of them is the
// counterpart allele (the alt base when the read shows the reference, the
// reference when it shows the alt), so that the bases agree with the alt
// counts of the read kernel.  Inserted bases draw their errors from the word
// mixed with their rank.  Indels anchored before p are not applied.
__device__ void build_read(const SeqParams& prm, const uint32_t* __restrict__ genome, const SeqRec* __restrict__ recs,
                           uint32_t n_recs, const uint32_t* __restrict__ aux, uint32_t p, uint32_t ce, uint32_t cell,
                           uint32_t inst, uint32_t w, uint32_t mate, SamRead& out, char* __restrict__ seq) {
  const char* ACGT = "ACGT";
  const uint32_t R = prm.read_len;
  const uint32_t wm = mate_word(w, mate);
  uint32_t i = lower_bound_rec(recs, n_recs, p);
  uint32_t q = p, n = 0, nc = 0;
  auto push = [&](uint32_t op, uint32_t len) {
    if (nc > 0 && (out.cigar[nc - 1] & 15u) == op) { out.cigar[nc - 1] += len << 4; return; }
    if (nc < SAM_MAX_CIGAR) out.cigar[nc++] = (len << 4) | op;
  };
  auto others = [](uint32_t tb, int first, uint32_t k) {   // k-th base other than tb (first: preferred one)
    uint32_t o[3] = {0, 0, 0}, m = 0;
    if (first >= 0 && uint32_t(first) != tb) o[m++] = uint32_t(first);
    for (uint32_t x = 0; x < 4 && m < 3; ++x) if (x != tb && (m == 0 || x != o[0])) o[m++] = x;
    return o[k];
  };
  bool indels_open = true;
  while (n < R && q < ce) {
    const uint32_t b = base_at(genome, q);
    while (i < n_recs && recs[i].locus < q) ++i;
    bool site = false, carried_snv = false;
    uint32_t alt = 0, indel = 0;
    bool has_indel = false;
    for (uint32_t k = i; k < n_recs && recs[k].locus == q; ++k) {
      const SeqRec r = recs[k];
      const bool carried = (r.tin <= cell) && (cell < r.tout) &&
                           inst_carries(prm, inst, r.info & 0xffffu, (uint64_t(r.tin) << 16) | ((r.info >> 16) & 0x7fffu));
      if (!(r.info >> 31)) {
        if (!site) { site = true; alt = aux[k] & 3u; }
        if (carried && !carried_snv) { carried_snv = true; alt = aux[k] & 3u; }
      } else if (carried && !has_indel) {
        has_indel = true;
        indel = aux[k];
      }
    }
    uint32_t tb = carried_snv ? alt : b;
    const uint32_t e = err_word(wm, q);
    if (e < prm.err_thr) tb = others(tb, site ? int(carried_snv ? b : alt) : -1, err_third(prm, e));
    // an unknown reference base (N) reads as N
    const bool unknown = prm.nmask && ((__ldg(prm.nmask + (q >> 5)) >> (q & 31u)) & 1u);
    seq[n++] = unknown ? 'N' : ACGT[tb];
    push(0u, 1u);
    ++q;
    if (has_indel && indels_open && nc < SAM_MAX_CIGAR - 2) {
      const uint32_t l = (indel >> 1) & 7u;
      if (indel & 1u) {
        for (uint32_t k = 0; k < l && n < R; ++k) {
          uint32_t ib = (indel >> (8 + 2 * k)) & 3u;
          const uint32_t ei = err_word(wm ^ (0x9E3779B1u * (k + 1)), q - 1);
          if (ei < prm.err_thr) ib = others(ib, -1, err_third(prm, ei));
          seq[n++] = ACGT[ib];
          push(1u, 1u);
        }
      } else if (n < R) {
        push(2u, l);
        q += l;
      }
    } else if (has_indel) {
      indels_open = false;       // the CIGAR is full: later indels are not applied
    }
  }
  out.pos = p;
  out.n_cigar = uint16_t(nc);
  out.seq_len = n;
}

__global__ void k_sam_reads(const SeqRec* __restrict__ recs, uint32_t n_recs, const uint32_t* __restrict__ aux,
                            const uint32_t* __restrict__ genome, SeqTiles tiles, uint32_t t0, uint32_t n_chunk,
                            const uint32_t* __restrict__ pair_cnt, const SeqSample* __restrict__ samples,
                            const uint32_t* __restrict__ leaf_tin, SeqParams prm, Key key,
                            const uint64_t* __restrict__ out_off, SamRead* __restrict__ out, char* __restrict__ seq,
                            uint32_t max_len) {
  const uint32_t k = blockIdx.x, s = blockIdx.y, t = t0 + k;
  const uint32_t n_pairs = pair_cnt[uint64_t(s) * tiles.n_tiles + t];
  const uint32_t start = tiles.start[t], len = tiles.len[t], ce = tiles.chr_end[t];
  const SeqSample sm = samples[s];
  const uint64_t base = out_off[uint64_t(s) * n_chunk + k];
  const uint32_t mates = prm.paired ? 2u : 1u;
  for (uint32_t j = threadIdx.x; j < n_pairs; j += blockDim.x) {
    const Fragment f = make_fragment<false>(key, j, t, s, start, len, ce, sm, leaf_tin, prm, nullptr);
    for (uint32_t m = 0; m < mates; ++m) {
      const uint64_t r = (base + j) * mates + m;
      SamRead& o = out[r];
      char* sq = seq + r * max_len;
      if (f.inst == 0xffffu) { o.pos = f.p0; o.mate_pos = f.p0; o.tlen = 0; o.flag = 4; o.n_cigar = 0; o.seq_len = 0; continue; }
      const uint32_t p = m ? f.p1 : f.p0;
      build_read(prm, genome, recs, n_recs, aux, p, ce, f.cell, f.inst, f.w, m, o, sq);
      if (prm.paired) {
        o.mate_pos = m ? f.p0 : f.p1;
        const int32_t span = int32_t(f.p1 + prm.read_len - f.p0);
        o.tlen = m ? -span : span;
        o.flag = uint16_t(0x1 | 0x2 | (m ? (0x80 | 0x10) : (0x40 | 0x20)));
      } else {
        o.mate_pos = 0; o.tlen = 0; o.flag = 0;
      }
    }
  }
}

void seq_sam_reads(const SeqRec* recs, uint32_t n_recs, const uint32_t* aux, const uint32_t* genome,
                   const SeqTiles& tiles, uint32_t t0, uint32_t n_chunk, const uint32_t* pair_cnt,
                   const SeqSample* samples, uint32_t n_samples, const uint32_t* leaf_tin, const SeqParams& prm,
                   uint64_t seed, const uint64_t* out_off, SamRead* out, char* seq, uint32_t max_len,
                   cudaStream_t st) {
  if (n_chunk == 0 || n_samples == 0) return;
  dim3 grid(n_chunk, n_samples);
  k_sam_reads<<<grid, 128, 0, st>>>(recs, n_recs, aux, genome, tiles, t0, n_chunk, pair_cnt, samples, leaf_tin, prm,
                                    make_key(seed), out_off, out, seq, max_len);
  note_launch();
}

// ------------------------------------------------------------ batched sequencing
__device__ __forceinline__ uint32_t batch_index(const uint32_t* __restrict__ off, uint32_t n, uint32_t x) {
  uint32_t lo = 0, hi = n;          // largest i < n with off[i] <= x
  while (hi - lo > 1) { const uint32_t mid = (lo + hi) >> 1; if (off[mid] <= x) lo = mid; else hi = mid; }
  return lo;
}

__global__ void k_seq_records_b(PlaceOut s, const uint16_t* __restrict__ inst_sorted, const uint32_t* __restrict__ n_dev,
                                uint32_t cap, SeqBatch b, SeqRec* __restrict__ recs) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= cap || i >= *n_dev) return;
  const uint32_t e = b.inst[inst_sorted[i]].etin_off + s.edge[i];
  SeqRec r;
  r.locus = s.locus[i];
  r.tin = b.etin[e];
  r.tout = b.etout[e];
  r.info = uint32_t(s.allele[i]) | ((uint32_t(s.seq[i]) & 0x7fffu) << 16) | (uint32_t(s.kind[i]) << 31);
  recs[i] = r;
}

__global__ void k_tile_ranges_b(SeqBatch b, const SeqRec* __restrict__ recs) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= b.n_tiles_all) return;
  const uint32_t i = b.tile_inst[t];
  const uint32_t r0 = b.rec_off[i], nr = b.rec_off[i + 1] - r0;
  const uint32_t start = b.tile_start[t];
  b.rec_lo[t] = lower_bound_rec(recs + r0, nr, start);
  b.rec_hi[t] = lower_bound_rec(recs + r0, nr, start + b.tile_len[t] - 1 + b.inst[i].prm.span);
}

__global__ void __launch_bounds__(SPLIT_THREADS) k_tile_counts_b(SeqBatch b) {
  const uint32_t gid = (blockIdx.x * SPLIT_THREADS + threadIdx.x) >> 5;   // one warp per block of tiles
  if (gid >= b.n_cnt) return;
  const uint32_t i = batch_index(b.cnt_off, b.n_inst, gid);
  const SeqInst& in = b.inst[i];
  const uint32_t local = gid - b.cnt_off[i], s = local / in.n_blocks, bi = in.blk_off + local % in.n_blocks;
  const uint32_t slot = in.slot_off + b.blk_slot[bi], first = b.c_first[slot];
  const TileSplit sp{b.c_nstarts[slot], in.T, b.c_ntiles[slot], nullptr, 0.0};
  tile_counts_warp(sp, s, b.blk_index[bi], b.c_depth[slot], b.c_id[slot], b.c_pairs[slot], b.keys[i],
                   b.pair_cnt + in.pair_off + uint64_t(s) * in.n_tiles + first);
}

// Read kernel of a batch: CTA (x, y, z) takes tile x of all the instances' tiles
// for the instance's sample y + z * gridDim.y, if it has that many.  (Resident CTAs that took
// items from a counter were no faster: 9.80 ms against 9.82 over 24 genomes.)
static_assert(sizeof(SeqParams) % 4 == 0 && sizeof(SeqParams) / 4 <= SEQ_THREADS, "SeqParams staging");

__global__ void __launch_bounds__(SEQ_THREADS, 4) k_reads_batch(SeqBatch b, const SeqRec* __restrict__ g_recs) {
  __shared__ __align__(16) ReadSmem sh;
  __shared__ SeqParams s_prm;
  const uint32_t gt = blockIdx.x, s = blockIdx.y + blockIdx.z * gridDim.y, i = b.tile_inst[gt];
  const SeqInst& in = b.inst[i];
  if (s >= in.n_samples) return;
  sh.s_hist[threadIdx.x] = make_uint4(0u, 0u, 0u, 0u);
  if (threadIdx.x < sizeof(SeqParams) / 4)
    reinterpret_cast<uint32_t*>(&s_prm)[threadIdx.x] = reinterpret_cast<const uint32_t*>(&in.prm)[threadIdx.x];
  const uint32_t t = gt - in.tile_off, lo = b.rec_lo[gt];
  const uint64_t rows = in.count_off + uint64_t(s) * in.count_stride;
  const SeqSample sm = b.samples[in.sample_off + s];
  const uint32_t n_pairs = b.pair_cnt[in.pair_off + uint64_t(s) * in.n_tiles + t];
  const SeqRec* recs = g_recs + b.rec_off[i];
  __syncthreads();
  read_tile(sh, recs, t, s, 0u, n_pairs, lo, b.rec_hi[gt] - lo, b.tile_start[gt], b.tile_len[gt], b.tile_end[gt], sm,
            b.leaf_tin, s_prm, b.keys[i], b.alt + rows, b.depth + rows);
}


// last atom starting at or before position a
__device__ __forceinline__ uint32_t atom_of(const uint32_t* __restrict__ atom_start, uint32_t n_atoms, uint32_t a) {
  uint32_t lo = 0, hi = n_atoms;
  while (hi - lo > 1) { const uint32_t mid = (lo + hi) >> 1; if (atom_start[mid] <= a) lo = mid; else hi = mid; }
  return lo;
}

__global__ void k_part_counts(uint32_t n_tiles, const uint32_t* __restrict__ tile_start,
                              const uint32_t* __restrict__ tile_len, const uint32_t* __restrict__ atom_start,
                              uint32_t n_atoms, uint32_t* __restrict__ cnt) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n_tiles) return;
  const uint32_t a = tile_start[t], b = a + tile_len[t];
  uint32_t x = atom_of(atom_start, n_atoms, a), n = 0;
  for (; x < n_atoms && atom_start[x] < b; ++x) ++n;
  cnt[t] = n;
}

__global__ void k_part_emit(uint32_t n_tiles, const uint32_t* __restrict__ tile_start,
                            const uint32_t* __restrict__ tile_len, const uint32_t* __restrict__ atom_start,
                            uint32_t n_atoms, uint32_t genome_len, const uint32_t* __restrict__ part_off,
                            uint32_t* __restrict__ part_start, uint32_t* __restrict__ part_len,
                            uint32_t* __restrict__ part_atom, uint32_t* __restrict__ tile_atom) {
  const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n_tiles) return;
  const uint32_t a = tile_start[t], b = a + tile_len[t];
  uint32_t q = part_off[t];
  for (uint32_t x = atom_of(atom_start, n_atoms, a); x < n_atoms && atom_start[x] < b; ++x, ++q) {
    const uint32_t lo = max(a, atom_start[x]);
    const uint32_t hi = min(b, x + 1 < n_atoms ? atom_start[x + 1] : genome_len);
    part_start[q] = lo; part_len[q] = hi - lo; part_atom[q] = x;
  }
  tile_atom[t] = q - part_off[t] == 1 ? part_atom[q - 1] : 0xffffffffu;
}

// mass of one stretch of starts with integer copy sums (i0, sum)
__device__ __forceinline__ double stretch_mass(double wn, double wt, uint64_t nl, uint64_t i0, uint64_t sum) {
  double m = wn * double(i0);
  if (nl > 0) m = m + (wt / double(nl)) * double(sum);
  return m;
}

// one thread per (sample, tile): the tile's mass and, for tiles of several
// parts, the thresholds floor(CDF * 2^31) of the part draw with the last
// part of positive mass at 2^31 (the host's cdf_thresholds)
__global__ void k_tile_mass(uint32_t n_samples, uint32_t n_tiles, const uint32_t* __restrict__ part_off,
                            const uint32_t* __restrict__ part_len, const uint32_t* __restrict__ part_atom,
                            uint32_t n_atoms, const double* __restrict__ wn_s, const double* __restrict__ wt_s,
                            const uint64_t* __restrict__ nl_s, const uint64_t* __restrict__ icnt0,
                            const uint64_t* __restrict__ copy_sum, uint32_t n_parts, uint64_t* __restrict__ tile_i0,
                            uint64_t* __restrict__ tile_s, uint32_t* __restrict__ part_cdf) {
  const uint64_t gid = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (gid >= uint64_t(n_samples) * n_tiles) return;
  const uint32_t s = uint32_t(gid / n_tiles), t = uint32_t(gid % n_tiles);
  const double wn = wn_s[s], wt = wt_s[s];
  const uint64_t nl = nl_s[s];
  const uint64_t* i0a = icnt0 + uint64_t(s) * n_atoms;
  const uint64_t* sa = copy_sum + uint64_t(s) * n_atoms;
  const uint32_t pb = part_off[t], pe = part_off[t + 1];
  uint64_t i0 = 0, sum = 0;
  for (uint32_t q = pb; q < pe; ++q) {
    const uint64_t len = part_len[q], x = part_atom[q];
    i0 += len * i0a[x];
    sum += len * sa[x];
  }
  if (pe - pb > 1) {
    double tot = 0.0;
    uint32_t last = pb;
    for (uint32_t q = pb; q < pe; ++q) {
      const uint64_t len = part_len[q], x = part_atom[q];
      const double w = stretch_mass(wn, wt, nl, len * i0a[x], len * sa[x]);
      tot += w;
      if (w > 0) last = q;
    }
    uint32_t* thr = part_cdf + uint64_t(s) * n_parts;
    double c = 0.0;
    for (uint32_t q = pb; q < pe; ++q) {
      const uint64_t len = part_len[q], x = part_atom[q];
      c += stretch_mass(wn, wt, nl, len * i0a[x], len * sa[x]);
      if (!(tot > 0)) { thr[q] = 0u; continue; }
      double v = floor(c / tot * 2147483648.0);
      if (v > 2147483648.0) v = 2147483648.0;
      thr[q] = (q >= last) ? 2147483648u : uint32_t(v);
    }
  }
  tile_i0[gid] = i0;
  tile_s[gid] = sum;
}

// one CTA per (sample, chromosome slot): the integer copy sums before each
// tile by an exclusive block scan (exact, so independent of the order of
// the additions), and the mass before each tile as the mass of those sums
constexpr uint32_t MASS_PER_THREAD = 4;
__global__ void __launch_bounds__(256) k_mass_prefix(uint32_t n_slots, const uint32_t* __restrict__ c_first,
                                                     const uint32_t* __restrict__ c_ntiles, uint32_t n_tiles,
                                                     const double* __restrict__ wn_s, const double* __restrict__ wt_s,
                                                     const uint64_t* __restrict__ nl_s,
                                                     const uint64_t* __restrict__ tile_i0,
                                                     const uint64_t* __restrict__ tile_s,
                                                     double* __restrict__ mass_cum, double* __restrict__ mass_tot) {
  __shared__ uint64_t w_i0[8], w_s[8];
  __shared__ uint64_t carry_i0, carry_s;
  const uint32_t s = blockIdx.x / n_slots, slot = blockIdx.x % n_slots;
  const uint32_t first = c_first[slot], nt = c_ntiles[slot];
  const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double wn = wn_s[s], wt = wt_s[s];
  const uint64_t nl = nl_s[s];
  const uint64_t base = uint64_t(s) * n_tiles + first;
  if (threadIdx.x == 0) { carry_i0 = 0; carry_s = 0; }
  __syncthreads();
  constexpr uint32_t CH = 256 * MASS_PER_THREAD;
  for (uint32_t c0 = 0; c0 < nt; c0 += CH) {
    uint64_t a[MASS_PER_THREAD], b[MASS_PER_THREAD], ta = 0, tb = 0;
#pragma unroll
    for (uint32_t q = 0; q < MASS_PER_THREAD; ++q) {
      const uint32_t t = c0 + threadIdx.x * MASS_PER_THREAD + q;
      a[q] = t < nt ? tile_i0[base + t] : 0;
      b[q] = t < nt ? tile_s[base + t] : 0;
      ta += a[q];
      tb += b[q];
    }
    // exclusive scan of the threads' sums: warp, then warps
    uint64_t ia = ta, ib = tb;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint64_t xa = __shfl_up_sync(0xffffffffu, ia, o), xb = __shfl_up_sync(0xffffffffu, ib, o);
      if (lane >= uint32_t(o)) { ia += xa; ib += xb; }
    }
    if (lane == 31) { w_i0[warp] = ia; w_s[warp] = ib; }
    __syncthreads();
    uint64_t pa = carry_i0, pb = carry_s;
    for (uint32_t w = 0; w < warp; ++w) { pa += w_i0[w]; pb += w_s[w]; }
    pa += ia - ta;
    pb += ib - tb;
#pragma unroll
    for (uint32_t q = 0; q < MASS_PER_THREAD; ++q) {
      const uint32_t t = c0 + threadIdx.x * MASS_PER_THREAD + q;
      if (t < nt) mass_cum[base + t] = stretch_mass(wn, wt, nl, pa, pb);
      pa += a[q];
      pb += b[q];
    }
    __syncthreads();
    if (threadIdx.x == 255) { carry_i0 = pa; carry_s = pb; }
    __syncthreads();
  }
  if (threadIdx.x == 0) mass_tot[uint64_t(s) * n_slots + slot] = stretch_mass(wn, wt, nl, carry_i0, carry_s);
}

void seq_tile_parts(uint32_t n_tiles, const uint32_t* tile_start, const uint32_t* tile_len,
                    const uint32_t* atom_start, uint32_t n_atoms, uint32_t genome_len, uint32_t* part_off,
                    uint32_t* scan_part, uint32_t* part_start, uint32_t* part_len, uint32_t* part_atom,
                    uint32_t* tile_atom, cudaStream_t st) {
  if (!n_tiles) return;
  k_part_counts<<<nblk(n_tiles), 256, 0, st>>>(n_tiles, tile_start, tile_len, atom_start, n_atoms, part_off);
  note_launch();
  scan_rows<uint32_t>(part_off, part_off, n_tiles, 1, scan_part, part_off + n_tiles, st);
  k_part_emit<<<nblk(n_tiles), 256, 0, st>>>(n_tiles, tile_start, tile_len, atom_start, n_atoms, genome_len,
                                             part_off, part_start, part_len, part_atom, tile_atom);
  note_launch();
}

void seq_tile_mass(uint32_t n_samples, uint32_t n_slots, const uint32_t* c_first, const uint32_t* c_ntiles,
                   const uint32_t* part_off, const uint32_t* part_len, const uint32_t* part_atom, uint32_t n_atoms,
                   const double* wn, const double* wt, const uint64_t* nl, const uint64_t* icnt0,
                   const uint64_t* copy_sum, uint32_t n_tiles, uint32_t n_parts, uint64_t* tile_sums,
                   double* mass_cum, double* mass_tot, uint32_t* part_cdf, cudaStream_t st) {
  const uint64_t n = uint64_t(n_samples) * n_tiles;
  if (!n) return;
  k_tile_mass<<<nblk(n), 256, 0, st>>>(n_samples, n_tiles, part_off, part_len, part_atom, n_atoms, wn, wt, nl, icnt0,
                                       copy_sum, n_parts, tile_sums, tile_sums + n, part_cdf);
  k_mass_prefix<<<n_samples * n_slots, 256, 0, st>>>(n_slots, c_first, c_ntiles, n_tiles, wn, wt, nl, tile_sums,
                                                     tile_sums + n, mass_cum, mass_tot);
  note_launch(2);
}

void seq_prepare(const SeqChroms& c, const SeqTiles& tiles, const PlaceOut& sorted, uint32_t n_recs,
                 const uint32_t* edge_tin, const uint32_t* edge_tout, uint32_t span, SeqRec* recs, uint32_t n_split,
                 uint64_t seed, uint32_t* pair_cnt, cudaStream_t st) {
  // (a split of more blocks than a grid has is launched on its own)
  const uint64_t split = uint64_t(n_split) * c.n_slots * split_blocks(c);
  const uint32_t rest = nblk(c.n_tiles, SPLIT_THREADS) + nblk(n_recs, SPLIT_THREADS);
  const bool apart = split + rest > MAX_GRID_X;
  if (apart) seq_tile_counts(c, n_split, nullptr, nullptr, seed, pair_cnt, st);
  const uint32_t split_end = apart ? 0u : uint32_t(split), tiles_end = split_end + nblk(c.n_tiles, SPLIT_THREADS);
  const uint32_t grid = split_end + rest;
  if (!grid) return;
  const Key key = make_key(seed);
  if (split_end)
    k_seq_prepare<true><<<grid, SPLIT_THREADS, 0, st>>>(c, tiles, sorted, n_recs, edge_tin, edge_tout, span, recs,
                                                        split_end, tiles_end, key, pair_cnt);
  else
    k_seq_prepare<false><<<grid, SPLIT_THREADS, 0, st>>>(c, tiles, sorted, n_recs, edge_tin, edge_tout, span, recs,
                                                         split_end, tiles_end, key, pair_cnt);
  note_launch();
}

void seq_tile_counts(const SeqChroms& c, uint32_t n_samples, const double* mass_cum, const double* mass_tot,
                     uint64_t seed, uint32_t* pair_cnt, cudaStream_t st) {
  // whole rows, as many at a time as a grid has blocks for
  const uint64_t rows = uint64_t(n_samples) * c.n_slots, per = split_blocks(c), most = MAX_GRID_X / std::max<uint64_t>(per, 1);
  for (uint64_t row = 0; per && row < rows; row += most) {
    const uint32_t grid = uint32_t(std::min(most, rows - row) * per);
    k_tile_split<<<grid, SPLIT_THREADS, 0, st>>>(c, row, mass_cum, mass_tot, make_key(seed), pair_cnt);
    note_launch();
  }
}

// ------------------------------------------------------------ observed rows
// The rows of the result a caller reads by default: mutations with an alt
// read in some sample (src/seq_simulation.cpp:52-90 keeps those unless
// include_non_sequenced_mutations).  Flags, their exclusive scan, then the
// compact [sample][row] tables and the rows' mutation indices.
__global__ void k_active_flags(const uint32_t* __restrict__ alt, uint32_t n_samples, uint64_t M,
                               uint32_t* __restrict__ flag) {
  const uint64_t m = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (m >= M) return;
  uint32_t any = 0;
  for (uint32_t s = 0; s < n_samples; ++s) any |= alt[uint64_t(s) * M + m];
  flag[m] = any ? 1u : 0u;
}

__global__ void k_active_gather(const uint32_t* __restrict__ alt, const uint32_t* __restrict__ depth,
                                uint32_t n_samples, uint64_t M, const uint32_t* __restrict__ pos, uint32_t n_active,
                                uint32_t* __restrict__ index, uint32_t* __restrict__ a_out,
                                uint32_t* __restrict__ d_out) {
  const uint64_t m = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (m >= M) return;
  const uint32_t p = pos[m];
  if ((m + 1 < M ? pos[m + 1] : n_active) == p) return;   // not observed
  index[p] = uint32_t(m);
  for (uint32_t s = 0; s < n_samples; ++s) {
    a_out[uint64_t(s) * n_active + p] = alt[uint64_t(s) * M + m];
    d_out[uint64_t(s) * n_active + p] = depth[uint64_t(s) * M + m];
  }
}

void seq_active_flags(const uint32_t* alt, uint32_t n_samples, uint64_t M, uint32_t* flag, cudaStream_t st) {
  if (M) { k_active_flags<<<nblk(M), 256, 0, st>>>(alt, n_samples, M, flag); note_launch(); }
}

void seq_active_gather(const uint32_t* alt, const uint32_t* depth, uint32_t n_samples, uint64_t M, const uint32_t* pos,
                       uint32_t n_active, uint32_t* index, uint32_t* a_out, uint32_t* d_out, cudaStream_t st) {
  if (M && n_active) {
    k_active_gather<<<nblk(M), 256, 0, st>>>(alt, depth, n_samples, M, pos, n_active, index, a_out, d_out);
    note_launch();
  }
}

void seq_reads(const SeqRec* recs, uint32_t n_recs, const SeqTiles& tiles, const uint32_t* pair_cnt,
               const SeqSample* samples, uint32_t n_samples, const uint32_t* leaf_tin, const SeqParams& prm,
               uint64_t seed, uint32_t* alt, uint32_t* depth, cudaStream_t st) {
  if (tiles.n_tiles == 0 || n_samples == 0 || n_recs == 0) return;
  dim3 grid(tiles.n_tiles, n_samples);
  const Key k = make_key(seed);
  k_reads<<<grid, SEQ_THREADS, 0, st>>>(recs, tiles, pair_cnt, samples, leaf_tin, prm, round_keys(k.k0, k.k1), n_recs,
                                         alt, depth); note_launch();
}

void seq_cn_rows(const SeqParams& prm, const SeqSample* samples, uint32_t n_samples, CnRow* rows, cudaStream_t st) {
  const uint64_t n = uint64_t(n_samples) * prm.n_atoms * SEQ_CN_OPTS;
  if (n) { k_cn_rows<<<nblk(n), 256, 0, st>>>(prm, samples, n_samples, rows); note_launch(); }
}

void seq_batch_records(const PlaceOut& sorted, const uint16_t* inst_sorted, const uint32_t* n_dev, uint32_t cap,
                       const SeqBatch& b, SeqRec* recs, cudaStream_t st) {
  if (cap) { k_seq_records_b<<<nblk(cap), 256, 0, st>>>(sorted, inst_sorted, n_dev, cap, b, recs); note_launch(); }
}

constexpr uint32_t MAX_GRID_YZ = 65535;
void seq_batch_reads(const SeqBatch& b, const SeqRec* recs, cudaStream_t st) {
  if (b.n_cnt) { k_tile_counts_b<<<nblk(uint64_t(b.n_cnt) * 32, SPLIT_THREADS), SPLIT_THREADS, 0, st>>>(b); note_launch(); }
  if (!b.n_tiles_all) return;
  k_tile_ranges_b<<<nblk(b.n_tiles_all), 256, 0, st>>>(b, recs); note_launch();
  if (b.max_samples) {
    const uint32_t z = (b.max_samples + MAX_GRID_YZ - 1) / MAX_GRID_YZ;
    k_reads_batch<<<dim3(b.n_tiles_all, (b.max_samples + z - 1) / z, z), SEQ_THREADS, 0, st>>>(b, recs); note_launch();
  }
}
}  // namespace pg
