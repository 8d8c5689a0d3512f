// Mutation placement on a samples forest.
//
// Reference call site: MutationEngine::place_mutations
// (src/mutation_engine.cpp:1085-1113) -> RACES
// MutationEngine<uint32_t, std::mt19937_64>::place_mutations (absent; model
// restated here and in oracle/).
//
// Model (one draw function per decision, all keyed Philox):
//   * edge v of the forest carries divisions d_v >= 1; division j happens at
//     t = t_parent + (t_v - t_parent) * (j+1)/d_v (roots: t_v), and belongs to
//     the exposure epoch whose start time is the last one <= t.
//   * passenger SNVs (indels) on (v, epoch e):
//       Poisson(rate[species_v][e] * allelic_size * divisions_in_e)
//     (per-species passenger rates: src/mutation_engine.cpp:864-1083; timed
//     exposures: :734-739).  The preneoplastic edge (index N) carries exactly
//     the requested numbers, drawn from the named signature
//     (src/mutation_engine.hpp:160-206).
//   * each mutation draws its signature from the epoch exposure, its class
//     from the signature, a position uniformly from the class's position list,
//     and an allele uniformly among the cell's alleles.
//   * infinite sites (src/mutation_engine.hpp:148-156): loci are unique over
//     the forest; colliding mutations keep their class and redraw the
//     position (attempt a uses Philox block 1+a), the lowest slot index wins
//     a contested locus, rounds repeat until no collision is left.  From
//     attempt RECLASS_ATTEMPTS on, the class is redrawn too (same signature),
//     so a class whose positions are all taken cannot stall the rounds.
#include <algorithm>

#include "pg_common.cuh"
#include "pg_rng.cuh"
#include "pg_fast.cuh"
#include "pg_scan.cuh"
#include "pg_kernels.h"

namespace pg {

constexpr uint32_t RECLASS_ATTEMPTS = 4;

// ------------------------------------------------------------ per-edge counts
__device__ __noinline__ uint64_t poisson_fp64(Stream st, double lambda) { return poisson(st, lambda); }
// poisson(st, lambda), in FP32 where that decides it
__device__ __forceinline__ uint64_t poisson_draw(const Stream& st, double lambda) {
  if (!(lambda > 0.0)) return 0;
  uint64_t k;
  return poisson_fast(st, lambda, k) ? k : poisson_fp64(st, lambda);
}

// divisions of edge v in each epoch: division j of d happens at
// tu + (tv - tu) ((j + 1) / d) and belongs to the last epoch started by then.
// Most edges lie within one epoch, which two comparisons per epoch show (the
// times stay within [tu, tv] up to rounding); the FP64 divisions of the
// others cost 330 ns each.
__device__ __forceinline__ void epoch_divisions(const PlaceTables& t, uint32_t v, uint32_t* ndiv) {
  const uint32_t E = t.n_epochs, d = t.divisions[v];
  for (uint32_t e = 0; e < E; ++e) ndiv[e] = 0;
  if (E == 1) { ndiv[0] = d; return; }
  const double tv = t.birth[v];
  const int par = t.parent[v];
  const double tu = par >= 0 ? t.birth[par] : tv;
  const double slack = double(fabsf(float(tu)) + fabsf(float(tv))) * 1e-9;
  const double lo = (tu < tv ? tu : tv) - slack, hi = (tu < tv ? tv : tu) + slack;
  uint32_t e0 = 0, e1 = 0;
  while (e0 + 1 < E && t.epoch_start[e0 + 1] <= lo) ++e0;
  e1 = e0;
  while (e1 + 1 < E && t.epoch_start[e1 + 1] <= hi) ++e1;
  if (e0 == e1) { ndiv[e0] = d; return; }
  for (uint32_t j = 0; j < d; ++j) {
    const double tj = tu + (tv - tu) * (double(j + 1) / double(d));
    uint32_t e = 0;
    while (e + 1 < E && t.epoch_start[e + 1] <= tj) ++e;
    ndiv[e] += 1;
  }
}

// counts of edge v (v == n_nodes: the preneoplastic edge), SNVs or indels,
// into cnt[v * n_epochs + e].  One thread per (edge, kind), drawing in FP32:
// 26 us for 6e4 edges (147 us with one thread per edge in FP64).
__device__ __forceinline__ void edge_counts_one(const PlaceTables& t, uint32_t v, bool indel, Key key,
                                                uint32_t* __restrict__ cnt, uint32_t n_pre) {
  const uint32_t N = t.n_nodes, E = t.n_epochs;
  cnt += uint64_t(v) * E;
  if (v == N) {  // preneoplastic edge
    for (uint32_t e = 0; e < E; ++e) cnt[e] = e == 0 ? n_pre : 0u;
    return;
  }
  const uint32_t sp = t.species[v];
  uint32_t ndiv[MAX_EPOCHS];
  epoch_divisions(t, v, ndiv);
  const double A = t.node_size[v];   // allelic size of the edge's genome
  const double* rate = (indel ? t.indel_rate : t.snv_rate) + sp * E;
  for (uint32_t e = 0; e < E; ++e) {
    uint32_t n = 0;
    if (ndiv[e]) n = uint32_t(poisson_draw(Stream{key, e, v, 0u, indel ? TAG_EDGE_INDEL : TAG_EDGE_SNV, 0u},
                                           rate[e] * A * double(ndiv[e])));
    cnt[e] = n;
  }
}

__global__ void __launch_bounds__(128) k_edge_counts(PlaceTables t, uint32_t* __restrict__ cnt_snv,
                                                     uint32_t* __restrict__ cnt_id, Key key, uint32_t n_pre_snv,
                                                     uint32_t n_pre_id) {
  const uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
  const bool indel = blockIdx.y != 0;
  if (v > t.n_nodes) return;
  edge_counts_one(t, v, indel, key, indel ? cnt_id : cnt_snv, indel ? n_pre_id : n_pre_snv);
}

// passenger CNA events per edge: Poisson(rate_cna[species] * 2G * divisions);
// the germline size is used so that the counts do not depend on the copy
// number the events themselves create
__global__ void k_cna_counts(PlaceTables t, uint32_t* __restrict__ cnt_cna, Key key, double germline_size) {
  const uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= t.n_nodes) return;
  const double lam = t.cna_rate[t.species[v]] * germline_size * double(t.divisions[v]);
  cnt_cna[v] = uint32_t(poisson_draw(Stream{key, 0u, v, 0u, TAG_EDGE_CNA, 0u}, lam));
}

// ------------------------------------------------------------ placement
__device__ __forceinline__ uint32_t find_cell(const uint32_t* __restrict__ off, uint32_t ncell, uint32_t i) {
  // largest q with off[q] <= i (off is the exclusive scan of the counts)
  uint32_t lo = 0, hi = ncell;
  while (hi - lo > 1) { const uint32_t mid = (lo + hi) >> 1; if (off[mid] <= i) lo = mid; else hi = mid; }
  return lo;
}

// The same for a whole warp of consecutive slots (i - lane the first; lanes
// past the end may repeat the last): a 32-way search for the first slot's
// cell, then the lanes rank themselves among the next 32 offsets: 4 or 5
// dependent loads where a search per lane takes 16 (60 000 cells).
__device__ __forceinline__ uint32_t find_cell_warp(const uint32_t* __restrict__ off, uint32_t ncell, uint32_t i) {
  constexpr uint32_t FULL = 0xffffffffu;
  const uint32_t lane = threadIdx.x & 31u, i0 = __shfl_sync(FULL, i, 0);
  uint32_t lo = 0, hi = ncell;                 // off[lo] <= i0 < off[hi]
  while (hi - lo > 1) {
    const uint32_t step = (hi - lo + 31) / 32, at = lo + (lane + 1) * step;
    const uint32_t below = __popc(__ballot_sync(FULL, at < hi && off[at] <= i0));   // (ascending: a run of lanes)
    lo += below * step;
    hi = min(hi, lo + step);
  }
  const uint32_t b = lo + 1 + lane < ncell ? off[lo + 1 + lane] : 0xffffffffu;
  if (__shfl_sync(FULL, b, 31) <= i0 + 31u) return lo + find_cell(off + lo, ncell - lo, i);
  uint32_t c = 0;                              // offsets at or below i
#pragma unroll
  for (uint32_t step = 16; step >= 1; step >>= 1)
    if (__shfl_sync(FULL, b, c + step - 1) <= i) c += step;
  return lo + c;
}

// A slot's mutation in unsorted order: its locus and a 16-byte record of the
// other columns (PlaceRaw), written once and gathered once by the sort.
__device__ __forceinline__ uint4 raw_record(uint32_t edge, uint32_t aux, uint32_t allele, uint32_t seq, uint32_t cls,
                                            uint32_t sig, uint32_t kind, uint32_t nature) {
  return make_uint4(edge, aux, allele | (seq << 16), cls | (sig << 8) | (kind << 16) | (nature << 24));
}

// Mutation m of (edge v, epoch e), SNV or indel
struct Mut {
  uint32_t v, e, m;
  bool is_id;
};

// The first words of a mutation: its signature (from the epoch's exposure)
// and class (from the signature).
__device__ __forceinline__ void draw_class(const PlaceTables& t, Key key, const Mut& u, uint32_t& cls, uint32_t& sig) {
  Stream st{key, u.m, u.v, u.e, u.is_id ? TAG_INDEL : TAG_SNV, 0u};
  const U4 r = st.next();
  const uint32_t row = (u.v == t.n_nodes) ? t.n_epochs : u.e;
  if (!u.is_id) {
    sig = cdf_lookup(t.sbs_expo_cdf + row * t.n_sbs_sigs, t.n_sbs_sigs, r.x);
    cls = cdf_lookup(t.sbs_sig_cdf + sig * N_SBS, N_SBS, r.y);
  } else {
    sig = cdf_lookup(t.id_expo_cdf + row * t.n_id_sigs, t.n_id_sigs, r.x);
    cls = cdf_lookup(t.id_sig_cdf + sig * N_ID, N_ID, r.y);
  }
}

// The site of attempt `attempt` (0: the first draw; its words depend on the
// mutation and the attempt alone): the position drawn from the class's list,
// the locus (LOCUS_INVALID where no allele of the edge's genome covers it)
// and the allele instance, uniform among the covering ones.  From attempt
// RECLASS_ATTEMPTS on the class is redrawn from the signature (its free
// positions may be exhausted).  False: the class has no positions.
struct Site {
  uint32_t p, locus, allele, cls, w;
};
// its position (locus: before the alleles are known; allele: the word that draws it)
__device__ __forceinline__ bool draw_position(const PlaceTables& t, Key key, const Mut& u, uint32_t attempt,
                                              uint32_t cls, uint32_t sig, Site& out) {
  Stream st{key, u.m, u.v, u.e, u.is_id ? TAG_INDEL : TAG_SNV, 1u + attempt};
  const U4 r = st.next();
  if (attempt >= RECLASS_ATTEMPTS)
    cls = u.is_id ? cdf_lookup(t.id_sig_cdf + sig * N_ID, N_ID, r.w) : cdf_lookup(t.sbs_sig_cdf + sig * N_SBS, N_SBS, r.w);
  const uint32_t list = u.is_id ? cls : uint32_t(sbs_class_context(int(cls)));
  const uint32_t len = u.is_id ? t.id_len[list] : t.ctx_len[list];
  if (len == 0) return false;
  const uint64_t j = uniform_index64(r.x, r.y, len);
  out.p = u.is_id ? t.id_lists[t.id_off[list] + j] : t.ctx_lists[t.ctx_off[list] + j];
  out.cls = cls;
  out.w = r.w;
  out.locus = u.is_id ? out.p - 1 : out.p;          // an indel's locus is its anchor base
  out.allele = r.z;
  return true;
}
// its allele among those of genotype class node_cls
__device__ __forceinline__ void draw_allele(const PlaceTables& t, uint32_t node_cls, Site& x) {
  if (t.gc.n_classes == 1) {                        // no copy-number events: instances 0 and 1 everywhere
    x.allele = uniform_index32(x.allele, 2u);
    return;
  }
  uint32_t ioff = 0;
  const uint32_t n = covering(t.gc, node_cls, x.locus, &ioff);
  if (n == 0) x.locus = LOCUS_INVALID;              // deleted here: redrawn
  else x.allele = t.gc.inst_list[ioff + uniform_index32(x.allele, n)];
}
__device__ __forceinline__ uint32_t node_class_of(const PlaceTables& t, uint32_t v) {
  return t.gc.n_classes == 1 ? 0u : t.gc.node_class[v];
}
__device__ __forceinline__ bool draw_site(const PlaceTables& t, Key key, const Mut& u, uint32_t attempt, uint32_t cls,
                                          uint32_t sig, Site& out) {
  if (!draw_position(t, key, u, attempt, cls, sig, out)) return false;
  draw_allele(t, node_class_of(t, u.v), out);
  return true;
}

// What a mutation of class cls at p (its locus, or the base after an indel's)
// does, from the bases there and its word w.  SNV: the alt base on the forward
// strand; indel: its descriptor (bit 0 insertion, bits 1-3 length, bits 8..
// inserted bases, 2 bits each).
__device__ __forceinline__ uint32_t site_aux(const uint32_t* __restrict__ genome, bool is_id, uint32_t p, uint32_t cls,
                                             uint32_t w) {
  const uint32_t ref = base_at(genome, p);
  if (!is_id) {
    const uint32_t alt_pyr = sbs_class_alt(int(cls));
    const bool fwd = (ref == 1u || ref == 3u);
    return fwd ? alt_pyr : 3u - alt_pyr;
  }
  uint32_t ins = 0, l = 1, bases = 0;
  if (cls < 12) { ins = 0; l = 1; }
  else if (cls < 24) {
    ins = 1; l = 1;
    const uint32_t idx = (cls - 12) % 6;
    if (idx >= 1) bases = ref;
    else bases = (cls < 18) ? ((w & 1u) ? 2u : 1u) : ((w & 1u) ? 0u : 3u);
  } else if (cls < 48) { ins = 0; l = (cls - 24) / 6 + 2; }
  else if (cls < 72) {
    ins = 1; l = (cls - 48) / 6 + 2;
    if ((cls - 48) % 6 >= 1) { for (uint32_t k = 0; k < l; ++k) bases |= base_at(genome, p + k) << (2 * k); }
    else bases = w & ((1u << (2 * l)) - 1u);
  } else {
    ins = 0; l = cls == 72 ? 2 : (cls < 75 ? 3 : (cls < 78 ? 4 : 5));
  }
  return ins | (l << 1) | (bases << 8);
}

// The slot's columns for site x.  The aux column holds the site's word for now:
// the gather after the sort looks up the bases, in locus order (here each would
// be a DRAM access of its own).
__device__ __forceinline__ void put_site(const PlaceTables& t, const PlaceRaw& o, uint32_t slot, const Mut& u,
                                         uint32_t sig, const Site& x) {
  const bool pre = u.v == t.n_nodes, ok = x.locus != LOCUS_INVALID;
  o.locus[slot] = x.locus;
  o.rec[slot] = raw_record(u.v, x.w, ok ? x.allele : 0u,
                           pre ? SEQ_PRENEOPLASTIC : SEQ_PASSENGER, x.cls, sig, u.is_id ? KIND_INDEL : KIND_SNV,
                           pre ? NATURE_PRENEOPLASTIC : NATURE_PASSENGER);
}

// The slots of one call (plain form: one instance) and of a batch.  Both give
// the mutation of a slot, found by a search over the (edge, epoch) cells for
// the first draw and from the edge of its record after that.
struct PlainSlots {
  PlaceTables t;
  Key k;
  const uint32_t *off_snv, *off_id;
  uint32_t n_snv;
  using Ref = uint32_t;      // (nothing to know beyond the slot)
  __device__ __forceinline__ const PlaceTables& tables(Ref) const { return t; }
  __device__ __forceinline__ Key key(Ref) const { return k; }
  // (a warp of consecutive slots; see find_cell_warp)
  __device__ __forceinline__ Mut first(uint32_t slot, Ref&) const {
    const bool is_id = slot >= n_snv;
    const uint32_t i = is_id ? slot - n_snv : slot, ncell = (t.n_nodes + 1) * t.n_epochs;
    const uint32_t* off = is_id ? off_id : off_snv;
    const bool one = __all_sync(0xffffffffu, is_id) || !__any_sync(0xffffffffu, is_id);   // the warp has one kind
    const uint32_t q = one ? find_cell_warp(off, ncell, i) : find_cell(off, ncell, i);
    return {q / t.n_epochs, q % t.n_epochs, i - off[q], is_id};
  }
  __device__ __forceinline__ Mut again(uint32_t slot, uint32_t edge, Ref&) const {
    const bool is_id = slot >= n_snv;
    const uint32_t i = is_id ? slot - n_snv : slot;
    const uint32_t* off = (is_id ? off_id : off_snv) + uint64_t(edge) * t.n_epochs;
    uint32_t e = 0;          // the last epoch of the edge that starts at or before i
    while (e + 1 < t.n_epochs && off[e + 1] <= i) ++e;
    return {edge, e, i - off[e], is_id};
  }
  // what the infinite-sites tables key a locus by
  using TabKey = uint32_t;
  __device__ __forceinline__ TabKey tab_key(uint32_t locus, Ref) const { return locus; }
};

// ------------------------------------------------------------ hash sets
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }
__device__ __forceinline__ uint32_t hash32(uint32_t k) {
  k ^= k >> 16; k *= 0x7feb352du; k ^= k >> 15; k *= 0x846ca68bu; k ^= k >> 16;
  return k;
}

// The first infinite-sites round over every slot, against one table of all
// its candidates: an entry is (locus << 32 | code), code 0 for a driver's
// locus and slot + 1 for a passenger's, and a locus keeps the smallest code.
// A passenger wins its locus when the entry holds its own code, i.e. when no
// driver and no smaller slot drew it: the rule of the later rounds (the
// smallest pending slot wins a free locus).  The table then holds exactly
// the taken loci (drivers and the round's winners), so the later rounds test
// it instead of inserting the winners into the accepted set.
// The losers are marked while inserting: a slot that finds a smaller code
// at its locus marks itself, one that replaces a larger code marks that
// code's slot, so every code but the final holder of each locus is marked.
constexpr unsigned long long FIRST_EMPTY = ~0ull;

__device__ __forceinline__ void first_insert(unsigned long long* __restrict__ tab, uint32_t mask, uint32_t k,
                                             uint32_t code, uint8_t* __restrict__ lost, uint32_t* __restrict__ err) {
  const unsigned long long mine = (static_cast<unsigned long long>(k) << 32) | code;
  uint32_t h = hash32(k) & mask;
  for (uint32_t probe = 0; probe <= mask; ++probe) {
    // the table is mostly empty: try the swap first (one round trip)
    const unsigned long long x = atomicCAS(tab + h, FIRST_EMPTY, mine);
    if (x == FIRST_EMPTY) return;
    if (uint32_t(x >> 32) == k) {
      unsigned long long old = x;
      if (x > mine) old = atomicMin(tab + h, mine);
      if (old < mine) {
        if (code) lost[code - 1] = 1;                     // a smaller code holds the locus
      } else if (old > mine) {
        const uint32_t oc = uint32_t(old);                // replaced: that code's slot loses
        if (oc) lost[oc - 1] = 1;
      }
      return;
    }
    h = (h + 1) & mask;
  }
  atomicOr(err, ERR_CAPACITY);
}

// the entry of locus k, or FIRST_EMPTY
__device__ __forceinline__ unsigned long long first_find(const unsigned long long* __restrict__ tab, uint32_t mask,
                                                         uint32_t k) {
  uint32_t h = hash32(k) & mask;
  for (uint32_t probe = 0; probe <= mask; ++probe) {
    const unsigned long long x = tab[h];
    if (x == FIRST_EMPTY || uint32_t(x >> 32) == k) return x;
    h = (h + 1) & mask;
  }
  return FIRST_EMPTY;
}

// the drivers' loci (the passengers' go in with their first draw, k_place_first)
__global__ void k_first_drivers(const uint32_t* __restrict__ drv_locus, uint32_t n_drv,
                                unsigned long long* __restrict__ tab, uint32_t mask, uint8_t* __restrict__ lost,
                                uint32_t* __restrict__ err) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n_drv) first_insert(tab, mask, drv_locus[i], 0u, lost, err);
}

// the marked slots, in no particular order (warp-aggregated appends)
// (one append per block of 256 slots)
__global__ void __launch_bounds__(256) k_first_collect(const uint8_t* __restrict__ lost, uint32_t n,
                                                       uint32_t* __restrict__ next, uint32_t* __restrict__ n_next) {
  __shared__ uint32_t s_cnt[8], s_base;
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const bool mine = i < n && lost[i];
  const uint32_t ballot = __ballot_sync(0xffffffffu, mine);
  if (lane == 0) s_cnt[warp] = __popc(ballot);
  __syncthreads();
  if (threadIdx.x == 0) {
    uint32_t tot = 0;
    for (int w = 0; w < 8; ++w) { const uint32_t c = s_cnt[w]; s_cnt[w] = tot; tot += c; }
    s_base = tot ? atomicAdd(n_next, tot) : 0u;
  }
  __syncthreads();
  if (mine) next[s_base + s_cnt[warp] + __popc(ballot & ((1u << lane) - 1u))] = i;
}

// The first draw of every slot.  With infinite sites its insertion into the
// first round's table is fused in: the insertion's atomics overlap the draws'
// gathers.  The drivers go in afterwards (k_first_drivers); the table's final
// state and the marks do not depend on the order of the insertions.  tab (all
// ones) and lost (zeros) are set by the caller.
// Bound by the latency of dependent loads, at full scale by random DRAM
// accesses (list entry, table entry): the cell by a search of the warp, the
// table's entry requested before the allele is looked up, the bases left to
// the gather after the sort.  35e6 slots on 3.1 Gbp: 2.82 -> 2.18 ms (the
// gather 0.72 -> 0.85); 1.75e6 on 155 Mbp: 120 -> 85 us.
__global__ void k_place_first(PlainSlots s, PlaceRaw o, uint32_t n_slots, unsigned long long* __restrict__ tab,
                              uint32_t mask, uint8_t* __restrict__ lost, uint32_t* __restrict__ err) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t ref = 0, cls, sig;
  const Mut u = s.first(min(i, n_slots - 1), ref);
  if (i >= n_slots) return;
  const uint32_t nc = node_class_of(s.t, u.v);
  draw_class(s.t, s.k, u, cls, sig);
  Site x;
  if (!draw_position(s.t, s.k, u, 0u, cls, sig, x)) { atomicOr(err, ERR_EMPTY_CLASS); o.locus[i] = 0; return; }
  if (tab) prefetch_l2(tab + (hash32(x.locus) & mask));
  draw_allele(s.t, nc, x);
  if (tab) {
    if (x.locus == LOCUS_INVALID) lost[i] = 1;           // no allele at the drawn position
    else first_insert(tab, mask, x.locus, i + 1, lost, err);
  }
  put_site(s.t, o, i, u, sig, x);
}

// ------------------------------------------------------------ redraws
// Colliding mutations redraw in rounds: in round r every pending slot proposes
// its attempt r; a locus goes to the smallest slot of the first round that
// proposes it, and the slots that did not get theirs propose again in round
// r + 1 (a locus taken in the first round, or without an allele, goes to
// nobody).  So a locus prefers the smallest (round, slot), each slot proposes
// its attempts in order, and the rounds are one execution of deferred
// acceptance (Gale and Shapley, "College admissions and the stability of
// marriage", Amer. Math. Monthly 69, 1962), whose outcome does not depend on
// the order of the proposals: a slot takes a locus from a holder that the
// locus likes less, and the displaced slot goes on with its next attempt.
// Each thread follows one proposer at a time, without rounds or barriers.
//
// A round used to cost three grid barriers or, with few slots pending, a block
// alone: 198 us for 3 x 1 Mbp (20 rounds, nearly all waiting), 1.36 ms at
// full scale.  Now the chain of the unluckiest slot bounds the small one and the
// gathers the large one: 25 us and 0.44 ms, both kernels.
template <class K> __device__ __forceinline__ K no_key() { return K(~K(0)); }
__device__ __forceinline__ uint32_t key_hash(uint32_t k) { return hash32(k); }
__device__ __forceinline__ uint64_t key_hash(uint64_t k) {
  k ^= k >> 33; k *= 0xff51afd7ed558ccdull; k ^= k >> 33; k *= 0xc4ceb9fe1a85ec53ull; k ^= k >> 33;
  return k;
}
__device__ __forceinline__ uint32_t key_cas(uint32_t* p, uint32_t k) { return atomicCAS(p, 0xffffffffu, k); }
__device__ __forceinline__ uint64_t key_cas(uint64_t* p, uint64_t k) {
  return atomicCAS(reinterpret_cast<unsigned long long*>(p), ~0ull, static_cast<unsigned long long>(k));
}
// entry of key k, inserted when absent (mask + 1 entries, a power of two)
template <class K>
__device__ __forceinline__ bool key_entry(K* __restrict__ keys, uint64_t mask, K k, uint64_t& h) {
  h = uint64_t(key_hash(k)) & mask;
  for (uint64_t probe = 0; probe <= mask; ++probe) {
    const K prev = key_cas(keys + h, k);
    if (prev == no_key<K>() || prev == k) return true;
    h = (h + 1) & mask;
  }
  return false;
}
constexpr unsigned long long SITE_FREE = ~0ull;   // holder: attempt << 32 | slot

__device__ __forceinline__ bool taken_first(const PlainSlots&, const unsigned long long* tab, uint64_t mask, uint32_t k) {
  return first_find(tab, uint32_t(mask), k) != FIRST_EMPTY;
}

// A slot that is given up (the call fails) gets a locus the sort can take.
__device__ __forceinline__ void give_up(const PlaceRaw& o, uint32_t slot, uint32_t* flags, uint32_t bit) {
  atomicOr(flags, bit);
  o.locus[slot] = 0;
}

// pending slots list[0 .. *n) (n <= cap, which sizes the grid)
template <class S, class First>
__global__ void __launch_bounds__(128) k_sites_settle(S s, PlaceRaw o, const uint32_t* __restrict__ list,
                                                      const uint32_t* __restrict__ n, const First* __restrict__ first,
                                                      uint64_t fmask, typename S::TabKey* __restrict__ keys,
                                                      unsigned long long* __restrict__ held, uint64_t mask,
                                                      TailCtl* __restrict__ ctl, uint32_t* __restrict__ err) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= *n) return;
  uint32_t slot = list[i], attempt = 1;
  for (;;) {
    const uint4 r = o.rec[slot];                // edge, and the first draw's class and signature
    typename S::Ref ref{};
    const Mut u = s.again(slot, r.x, ref);
    const PlaceTables& t = s.tables(ref);
    const Key key = s.key(ref);
    for (;; ++attempt) {                        // the slot's next attempt at a locus that is not taken
      if (attempt >= TAIL_MAX_ROUND) { give_up(o, slot, &ctl->status, TAIL_ROUNDS_EXHAUSTED); return; }
      Site x;
      if (!draw_site(t, key, u, attempt, r.w & 0xffu, (r.w >> 8) & 0xffu, x)) {
        give_up(o, slot, err, ERR_EMPTY_CLASS);
        return;
      }
      if (x.locus == LOCUS_INVALID) continue;
      const typename S::TabKey k = s.tab_key(x.locus, ref);
      if (taken_first(s, first, fmask, k)) continue;
      uint64_t h;
      if (!key_entry(keys, mask, k, h)) { give_up(o, slot, err, ERR_CAPACITY); return; }
      const unsigned long long mine = (static_cast<unsigned long long>(attempt) << 32) | slot;
      const unsigned long long old = atomicMin(held + h, mine);
      if (old == SITE_FREE) return;
      if (old > mine) {                         // the holder is displaced: go on with it
        slot = uint32_t(old);
        attempt = uint32_t(old >> 32) + 1;
        break;
      }
    }
  }
}

// every settled slot's columns, from the table of holders
template <class S>
__global__ void __launch_bounds__(256) k_sites_final(S s, PlaceRaw o, const unsigned long long* __restrict__ held,
                                                     uint64_t cap, TailCtl* __restrict__ ctl,
                                                     uint32_t* __restrict__ err) {
  const uint64_t h = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  const unsigned long long w = h < cap ? held[h] : SITE_FREE;
  uint32_t attempt = 0;
  if (w != SITE_FREE) {
    const uint32_t slot = uint32_t(w);
    attempt = uint32_t(w >> 32);
    const uint4 r = o.rec[slot];
    typename S::Ref ref{};
    const Mut u = s.again(slot, r.x, ref);
    const uint32_t sig = (r.w >> 8) & 0xffu;
    Site x;
    if (!draw_site(s.tables(ref), s.key(ref), u, attempt, r.w & 0xffu, sig, x)) give_up(o, slot, err, ERR_EMPTY_CLASS);
    else put_site(s.tables(ref), o, slot, u, sig, x);
  }
  attempt = __reduce_max_sync(0xffffffffu, attempt);
  if ((threadIdx.x & 31u) == 0 && attempt) atomicMax(&ctl->rounds, attempt + 1);
}

// Without infinite sites: slots whose first draw lies where the cell has no
// allele left take their next attempt at a locus that has one.
__global__ void __launch_bounds__(128) k_sites_covered(PlainSlots s, PlaceRaw o, uint32_t n_slots,
                                                       TailCtl* __restrict__ ctl, uint32_t* __restrict__ err) {
  const uint32_t slot = blockIdx.x * blockDim.x + threadIdx.x;
  if (slot >= n_slots) return;
  uint32_t attempt = 0;
  if (o.locus[slot] == LOCUS_INVALID) {
    const uint4 r = o.rec[slot];
    uint32_t ref = 0;
    const Mut u = s.again(slot, r.x, ref);
    const uint32_t sig = (r.w >> 8) & 0xffu;
    Site x;
    do {
      if (++attempt >= TAIL_MAX_ROUND) { give_up(o, slot, &ctl->status, TAIL_ROUNDS_EXHAUSTED); return; }
      if (!draw_site(s.t, s.k, u, attempt, r.w & 0xffu, sig, x)) { give_up(o, slot, err, ERR_EMPTY_CLASS); return; }
    } while (x.locus == LOCUS_INVALID);
    put_site(s.t, o, slot, u, sig, x);
  }
  if (attempt || slot == 0) atomicMax(&ctl->rounds, attempt + 1);
}

// ------------------------------------------------------------ drivers
// Driver SIDs are applied on the first edge of their mutant, in application
// order with the mutant's CNAs and WGDs; their instance and order on the edge
// come from the host, which replays those events.
__global__ void k_drivers(PlaceRaw o, const DriverRec* __restrict__ drv, uint32_t n_drv, uint32_t base_slot) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_drv) return;
  const DriverRec d = drv[i];
  const uint32_t slot = base_slot + i;
  o.locus[slot] = d.locus;
  o.rec[slot] = raw_record(d.edge, d.aux, d.allele & 0xffffu, d.seq & 0xffffu, 0xffu, 0xffu, d.kind, NATURE_DRIVER);
}

// ------------------------------------------------------------ locus sort
constexpr int BUCKET_SHIFT = 10;

// Whether slots were given up: the call fails, and nothing is sorted (they all
// hold locus 0, and one thread would sort their bucket by insertion).
__device__ __forceinline__ bool failed(const PlaceFlags& f) {
  return *f.err != 0u || (f.tail && f.tail->status != 0u);
}

__global__ void k_bucket_count(const uint32_t* __restrict__ locus, uint32_t n, uint32_t* __restrict__ bcnt,
                               PlaceFlags flags) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n && !failed(flags)) atomicAdd(bcnt + (locus[i] >> BUCKET_SHIFT), 1u);
}
// Bucket sort on 64-bit keys (locus << 32 | slot) written by the scatter:
// the in-bucket insertion sort reads its bucket's keys contiguously, and
// ties of a locus fall in slot order.
__global__ void k_bucket_scatter_keys(const uint32_t* __restrict__ locus, uint32_t n, const uint32_t* __restrict__ boff,
                                      uint32_t* __restrict__ bfill, unsigned long long* __restrict__ keys,
                                      PlaceFlags flags) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || failed(flags)) return;
  const uint32_t k = locus[i], b = k >> BUCKET_SHIFT;
  keys[boff[b] + atomicAdd(bfill + b, 1u)] = (static_cast<unsigned long long>(k) << 32) | i;
}
// One block per 64 consecutive buckets: their keys (one contiguous range) are
// staged in shared memory and each thread ranks one key at a time in its
// bucket (a bucket holds a dozen keys at the usual densities), then writes the
// sorted locus and slot.  (With one thread insertion-sorting each bucket the
// kernel took 16 us for 35,000 keys and 375 us for 3.5e7.)  A range larger
// than the stage is sorted in place in global memory, a thread per bucket.
constexpr uint32_t SORT_BUCKETS = 64, SORT_STAGE = 2560, SORT_THREADS = 256;   // 20 KB of keys

__global__ void __launch_bounds__(SORT_THREADS) k_bucket_sort_keys(const uint32_t* __restrict__ boff, uint32_t nb,
                                                                   uint32_t n, unsigned long long* __restrict__ keys,
                                                                   uint32_t* __restrict__ locus,
                                                                   uint32_t* __restrict__ order, PlaceFlags flags) {
  __shared__ unsigned long long s_keys[SORT_STAGE];
  __shared__ uint32_t s_off[SORT_BUCKETS + 1];
  if (failed(flags)) return;
  const uint32_t b0 = blockIdx.x * SORT_BUCKETS, b1 = min(b0 + SORT_BUCKETS, nb), m = b1 - b0;
  if (threadIdx.x <= m) s_off[threadIdx.x] = b0 + threadIdx.x < nb ? boff[b0 + threadIdx.x] : n;
  __syncthreads();
  const uint32_t k0 = s_off[0], k1 = s_off[m];
  if (k1 - k0 <= SORT_STAGE) {
    for (uint32_t i = k0 + threadIdx.x; i < k1; i += SORT_THREADS) s_keys[i - k0] = keys[i];
    __syncthreads();
    for (uint32_t i = k0 + threadIdx.x; i < k1; i += SORT_THREADS) {
      uint32_t lo = 0, hi = m;                              // the bucket of key i
      while (hi - lo > 1) { const uint32_t mid = (lo + hi) >> 1; if (s_off[mid] <= i) lo = mid; else hi = mid; }
      const unsigned long long key = s_keys[i - k0];
      uint32_t at = s_off[lo];
      for (uint32_t j = s_off[lo] - k0; j < s_off[lo + 1] - k0; ++j) at += s_keys[j] < key ? 1u : 0u;
      locus[at] = uint32_t(key >> 32);
      order[at] = uint32_t(key);
    }
  } else if (threadIdx.x < m) {
    const uint32_t lo = s_off[threadIdx.x], hi = s_off[threadIdx.x + 1];
    for (uint32_t i = lo + 1; i < hi; ++i) {
      const unsigned long long kx = keys[i];
      uint32_t j = i;
      while (j > lo) {
        const unsigned long long ky = keys[j - 1];
        if (ky <= kx) break;
        keys[j] = ky;
        --j;
      }
      keys[j] = kx;
    }
    for (uint32_t i = lo; i < hi; ++i) { locus[i] = uint32_t(keys[i] >> 32); order[i] = uint32_t(keys[i]); }
  }
}

// The sorted columns: one 16-byte record per mutation, a passenger's aux from
// the bases at its locus (drivers bring theirs).
// (n_inst: a batch, whose instance i starts at boff[i * nb]; else 0)
__global__ void k_gather_records(const uint4* __restrict__ rec, const uint32_t* __restrict__ order, uint32_t n,
                                 const uint32_t* __restrict__ genome, PlaceOut s, uint16_t* __restrict__ inst_sorted,
                                 uint32_t n_inst, uint32_t nb, const uint32_t* __restrict__ boff, PlaceFlags flags) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || failed(flags)) return;
  const uint4 a = rec[order[i]];
  const bool is_id = ((a.w >> 16) & 0xffu) == KIND_INDEL;
  s.edge[i] = a.x;
  s.aux[i] = a.w >> 24 == NATURE_DRIVER ? a.y
                                        : site_aux(genome, is_id, s.locus[i] + (is_id ? 1u : 0u), a.w & 0xffu, a.y);
  s.allele[i] = uint16_t(a.z); s.seq[i] = uint16_t(a.z >> 16);
  s.cls[i] = uint8_t(a.w); s.sig[i] = uint8_t(a.w >> 8); s.kind[i] = uint8_t(a.w >> 16); s.nature[i] = uint8_t(a.w >> 24);
  if (n_inst) {
    uint32_t lo = 0, hi = n_inst;
    while (hi - lo > 1) { const uint32_t mid = (lo + hi) >> 1; if (boff[uint64_t(mid) * nb] <= i) lo = mid; else hi = mid; }
    inst_sorted[i] = uint16_t(lo);
  }
}

// ------------------------------------------------------------ batched placement
// A batch places the forests of many instances on one genome in single
// launches.  Cells (edge, epoch) of instance i occupy [cell_off[i],
// cell_off[i+1]) of the count arrays; the global slot space is every SNV of
// every instance (cells in order) followed by every indel, so the slots of
// one instance keep their relative order and every per-instance decision
// (Philox counters, lowest-slot wins, ties of the sort) is that of the plain
// path for the instance alone.
__device__ __forceinline__ uint32_t upper_index(const uint32_t* __restrict__ off, uint32_t n, uint32_t x) {
  // largest i < n with off[i] <= x
  uint32_t lo = 0, hi = n;
  while (hi - lo > 1) { const uint32_t mid = (lo + hi) >> 1; if (off[mid] <= x) lo = mid; else hi = mid; }
  return lo;
}

__global__ void k_edge_counts_b(const PlaceTables* __restrict__ tabs, uint32_t n_inst,
                                const uint32_t* __restrict__ node_off, const uint32_t* __restrict__ cell_off,
                                const Key* __restrict__ keys, const uint32_t* __restrict__ pre_snv,
                                const uint32_t* __restrict__ pre_id, uint32_t* __restrict__ cnt_snv,
                                uint32_t* __restrict__ cnt_id) {
  const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
  const bool indel = blockIdx.y != 0;
  if (g >= node_off[n_inst]) return;
  const uint32_t i = upper_index(node_off, n_inst, g);
  edge_counts_one(tabs[i], g - node_off[i], indel, keys[i], (indel ? cnt_id : cnt_snv) + cell_off[i],
                  (indel ? pre_id : pre_snv)[i]);
}

struct BatchSlots {
  const PlaceTables* tabs;
  const Key* keys;
  uint32_t n_inst;
  const uint32_t* cell_off;
  uint16_t* inst_of;
  const uint32_t *off_snv, *off_id;
  uint32_t n_snv;
  using Ref = uint32_t;      // the instance
  __device__ __forceinline__ const PlaceTables& tables(Ref i) const { return tabs[i]; }
  __device__ __forceinline__ Key key(Ref i) const { return keys[i]; }
  __device__ __forceinline__ Mut first(uint32_t slot, Ref& inst) const {
    const bool is_id = slot >= n_snv;
    const uint32_t j = is_id ? slot - n_snv : slot, ncell = cell_off[n_inst];
    const uint32_t* off = is_id ? off_id : off_snv;
    const bool one = __all_sync(0xffffffffu, is_id) || !__any_sync(0xffffffffu, is_id);   // the warp has one kind
    const uint32_t q = one ? find_cell_warp(off, ncell, j) : find_cell(off, ncell, j);    // global cell
    inst = upper_index(cell_off, n_inst, q);
    const uint32_t lq = q - cell_off[inst], E = tabs[inst].n_epochs;
    return {lq / E, lq % E, j - off[q], is_id};
  }
  __device__ __forceinline__ Mut again(uint32_t slot, uint32_t edge, Ref& inst) const {
    const bool is_id = slot >= n_snv;
    const uint32_t j = is_id ? slot - n_snv : slot;
    inst = inst_of[slot];
    const uint32_t E = tabs[inst].n_epochs;
    const uint32_t* off = (is_id ? off_id : off_snv) + cell_off[inst] + edge * E;
    uint32_t e = 0;
    while (e + 1 < E && off[e + 1] <= j) ++e;
    return {edge, e, j - off[e], is_id};
  }
  // loci are unique per instance
  using TabKey = uint64_t;
  __device__ __forceinline__ TabKey tab_key(uint32_t locus, Ref inst) const { return (uint64_t(inst) << 32) | locus; }
};

// the first round's table of a batch: its keys
__device__ __forceinline__ bool taken_first(const BatchSlots&, const uint64_t* keys, uint64_t mask, uint64_t k) {
  uint64_t h = key_hash(k) & mask;
  for (uint64_t probe = 0; probe <= mask; ++probe) {
    const uint64_t x = keys[h];
    if (x == k) return true;
    if (x == no_key<uint64_t>()) return false;
    h = (h + 1) & mask;
  }
  return false;
}

// The first draw of every slot of a batch and, with infinite sites (fkeys not
// NULL), its insertion into the first round's table, the losers marked as in
// the plain form: a slot that finds a smaller one at its locus, or that a
// smaller one replaces.
__global__ void k_place_first_b(BatchSlots s, PlaceRaw o, uint32_t n_slots, uint64_t* __restrict__ fkeys,
                                uint32_t* __restrict__ fslot, uint64_t fmask, uint8_t* __restrict__ lost,
                                uint32_t* __restrict__ err) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t inst, cls, sig;
  const Mut u = s.first(min(i, n_slots - 1), inst);
  if (i >= n_slots) return;
  const PlaceTables& t = s.tabs[inst];
  const Key key = s.keys[inst];
  s.inst_of[i] = uint16_t(inst);
  draw_class(t, key, u, cls, sig);
  Site x;
  if (!draw_position(t, key, u, 0u, cls, sig, x)) { atomicOr(err, ERR_EMPTY_CLASS); o.locus[i] = 0; return; }
  uint64_t h = 0;
  if (fkeys) {
    h = key_hash(s.tab_key(x.locus, inst)) & fmask;
    prefetch_l2(fkeys + h);
    prefetch_l2(fslot + h);
  }
  draw_allele(t, node_class_of(t, u.v), x);
  if (fkeys) {
    if (x.locus == LOCUS_INVALID) {
      lost[i] = 1;
    } else if (!key_entry(fkeys, fmask, s.tab_key(x.locus, inst), h)) {
      atomicOr(err, ERR_CAPACITY);
    } else {
      const uint32_t old = atomicMin(fslot + h, i);
      if (old < i) lost[i] = 1;
      else if (old != 0xffffffffu) lost[old] = 1;
    }
  }
  put_site(t, o, i, u, sig, x);
}

// sort of a batch by (instance, locus): bucket = instance * nb + locus >> 10
__global__ void k_bucket_count_b(const uint32_t* __restrict__ locus, const uint16_t* __restrict__ inst_of, uint32_t n,
                                 uint32_t nb, uint32_t* __restrict__ bcnt, PlaceFlags flags) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n && !failed(flags)) atomicAdd(bcnt + uint64_t(inst_of[i]) * nb + (locus[i] >> BUCKET_SHIFT), 1u);
}
__global__ void k_bucket_scatter_b(const uint32_t* __restrict__ locus, const uint16_t* __restrict__ inst_of,
                                   uint32_t n, uint32_t nb, const uint32_t* __restrict__ boff,
                                   uint32_t* __restrict__ bfill, unsigned long long* __restrict__ keys,
                                   PlaceFlags flags) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n || failed(flags)) return;
  const uint32_t k = locus[i];
  const uint64_t b = uint64_t(inst_of[i]) * nb + (k >> BUCKET_SHIFT);
  keys[boff[b] + atomicAdd(bfill + b, 1u)] = (static_cast<unsigned long long>(k) << 32) | i;
}

// ------------------------------------------------------------ host launchers
static inline unsigned nblk(uint64_t n, int b = 256) { return unsigned((n + b - 1) / b); }

void place_cna_counts(const PlaceTables& t, uint32_t* cnt_cna, uint64_t seed, double germline_size, cudaStream_t st) {
  if (t.n_nodes) { k_cna_counts<<<nblk(t.n_nodes, 128), 128, 0, st>>>(t, cnt_cna, make_key(seed), germline_size); note_launch(); }
}

void place_edge_counts(const PlaceTables& t, uint32_t* cnt_snv, uint32_t* cnt_id, uint64_t seed,
                       uint32_t n_pre_snv, uint32_t n_pre_id, cudaStream_t st) {
  k_edge_counts<<<dim3(nblk(t.n_nodes + 1, 128), 2), 128, 0, st>>>(t, cnt_snv, cnt_id, make_key(seed), n_pre_snv, n_pre_id);
  note_launch();
}

void place_drivers(const PlaceRaw& o, const DriverRec* drv, uint32_t n_drv, uint32_t base_slot, cudaStream_t st) {
  if (n_drv == 0) return;
  k_drivers<<<nblk(n_drv), 256, 0, st>>>(o, drv, n_drv, base_slot); note_launch();
}

void place_first_round(const PlaceTables& t, const PlaceRaw& o, uint64_t seed, const uint32_t* off_snv,
                       const uint32_t* off_id, uint32_t n_snv, uint32_t n_slots, unsigned long long* first,
                       uint32_t fmask, uint8_t* lost, uint32_t* err, cudaStream_t st) {
  if (n_slots == 0) return;
  if (first) cudaMemsetAsync(lost, 0, n_slots, st);
  k_place_first<<<nblk(n_slots), 256, 0, st>>>(PlainSlots{t, make_key(seed), off_snv, off_id, n_snv}, o, n_slots,
                                               first, fmask, lost, err);
  note_launch();
}

void sites_first_finish(const uint32_t* drv_locus, uint32_t n_drv, unsigned long long* first, uint32_t fmask,
                        uint8_t* lost, uint32_t n_slots, uint32_t* next, uint32_t* n_next, uint32_t* err,
                        cudaStream_t st) {
  if (n_drv) {
    k_first_drivers<<<nblk(n_drv), 256, 0, st>>>(drv_locus, n_drv, first, fmask, lost, err);
    note_launch();
  }
  if (n_slots) { k_first_collect<<<nblk(n_slots), 256, 0, st>>>(lost, n_slots, next, n_next); note_launch(); }
}

void sites_settle(const PlaceTables& t, const PlaceRaw& o, uint64_t seed, const uint32_t* off_snv,
                  const uint32_t* off_id, uint32_t n_snv, const uint32_t* list, const uint32_t* n, uint32_t n_max,
                  const unsigned long long* first, uint32_t fmask, uint32_t* keys, unsigned long long* held,
                  uint64_t cap, TailCtl* ctl, uint32_t* err, cudaStream_t st) {
  if (n_max == 0) return;
  const PlainSlots s{t, make_key(seed), off_snv, off_id, n_snv};
  k_sites_settle<<<nblk(n_max, 128), 128, 0, st>>>(s, o, list, n, first, uint64_t(fmask), keys, held, cap - 1, ctl, err);
  k_sites_final<<<nblk(cap), 256, 0, st>>>(s, o, held, cap, ctl, err);
  note_launch(2);
}

void sites_covered(const PlaceTables& t, const PlaceRaw& o, uint64_t seed, const uint32_t* off_snv,
                   const uint32_t* off_id, uint32_t n_snv, uint32_t n_slots, TailCtl* ctl, uint32_t* err,
                   cudaStream_t st) {
  if (n_slots == 0) return;
  k_sites_covered<<<nblk(n_slots, 128), 128, 0, st>>>(PlainSlots{t, make_key(seed), off_snv, off_id, n_snv}, o,
                                                      n_slots, ctl, err);
  note_launch();
}

void sort_by_locus(const PlaceRaw& o, uint32_t n, const uint32_t* genome, uint64_t G, uint32_t* bcnt, uint32_t* part,
                   uint32_t* order, const PlaceOut& sorted, unsigned long long* keys, const PlaceFlags& flags, cudaStream_t st) {
  const uint32_t nb = uint32_t((G >> BUCKET_SHIFT) + 1);
  uint32_t* const bfill = bcnt + nb;
  cudaMemsetAsync(bcnt, 0, sizeof(uint32_t) * 2 * nb, st);
  if (n == 0) return;
  k_bucket_count<<<nblk(n), 256, 0, st>>>(o.locus, n, bcnt, flags); note_launch();
  scan_rows<uint32_t>(bcnt, bcnt, nb, 1, part, nullptr, st);
  k_bucket_scatter_keys<<<nblk(n), 256, 0, st>>>(o.locus, n, bcnt, bfill, keys, flags); note_launch();
  k_bucket_sort_keys<<<nblk(nb, SORT_BUCKETS), SORT_THREADS, 0, st>>>(bcnt, nb, n, keys, sorted.locus, order, flags);
  k_gather_records<<<nblk(n), 256, 0, st>>>(o.rec, order, n, genome, sorted, nullptr, 0u, 0u, nullptr, flags);
  note_launch(2);
}

uint32_t sort_num_buckets(uint64_t G) { return uint32_t((G >> BUCKET_SHIFT) + 1); }

void place_edge_counts_batch(const PlaceTables* tabs, uint32_t n_inst, const uint32_t* node_off, uint32_t n_nodes_all,
                             const uint32_t* cell_off, const Key* keys, const uint32_t* pre_snv, const uint32_t* pre_id,
                             uint32_t* cnt_snv, uint32_t* cnt_id, cudaStream_t st) {
  if (n_nodes_all) {
    k_edge_counts_b<<<dim3(nblk(n_nodes_all, 128), 2), 128, 0, st>>>(tabs, n_inst, node_off, cell_off, keys, pre_snv,
                                                                     pre_id, cnt_snv, cnt_id);
    note_launch();
  }
}

void place_first_round_batch(const PlaceTables* tabs, uint32_t n_inst, const uint32_t* cell_off, const Key* keys,
                             const PlaceRaw& o, uint16_t* inst_of, const uint32_t* off_snv, const uint32_t* off_id,
                             uint32_t n_snv, uint32_t n_slots, uint64_t* fkeys, uint32_t* fslot, uint64_t fmask,
                             uint8_t* lost, uint32_t* next, uint32_t* n_next, uint32_t* err, cudaStream_t st) {
  if (n_slots == 0) return;
  if (fkeys) cudaMemsetAsync(lost, 0, n_slots, st);
  k_place_first_b<<<nblk(n_slots), 256, 0, st>>>(BatchSlots{tabs, keys, n_inst, cell_off, inst_of, off_snv, off_id, n_snv},
                                                 o, n_slots, fkeys, fslot, fmask, lost, err);
  note_launch();
  if (fkeys) { k_first_collect<<<nblk(n_slots), 256, 0, st>>>(lost, n_slots, next, n_next); note_launch(); }
}

void sites_settle_batch(const PlaceTables* tabs, uint32_t n_inst, const uint32_t* cell_off, const Key* keys,
                        const PlaceRaw& o, uint16_t* inst_of, const uint32_t* off_snv, const uint32_t* off_id,
                        uint32_t n_snv, const uint32_t* list, const uint32_t* n, uint32_t n_max, const uint64_t* fkeys,
                        uint64_t fmask, uint64_t* hkeys, unsigned long long* held, uint64_t cap, TailCtl* ctl,
                        uint32_t* err, cudaStream_t st) {
  if (n_max == 0) return;
  const BatchSlots s{tabs, keys, n_inst, cell_off, inst_of, off_snv, off_id, n_snv};
  k_sites_settle<<<nblk(n_max, 128), 128, 0, st>>>(s, o, list, n, fkeys, fmask, hkeys, held, cap - 1, ctl, err);
  k_sites_final<<<nblk(cap), 256, 0, st>>>(s, o, held, cap, ctl, err);
  note_launch(2);
}

void sort_batch(const PlaceRaw& o, const uint16_t* inst_of, uint32_t n, uint32_t n_inst, const uint32_t* genome,
                uint64_t G, uint32_t* bcnt, uint32_t* bfill, uint32_t* part, uint32_t* order, const PlaceOut& sorted, uint16_t* inst_sorted,
                unsigned long long* keys, const PlaceFlags& flags, cudaStream_t st) {
  const uint32_t nb = uint32_t((G >> BUCKET_SHIFT) + 1);
  const uint64_t nbt = uint64_t(nb) * n_inst;
  cudaMemsetAsync(bcnt, 0, sizeof(uint32_t) * (nbt + 1), st);
  cudaMemsetAsync(bfill, 0, sizeof(uint32_t) * nbt, st);
  if (n == 0) return;
  k_bucket_count_b<<<nblk(n), 256, 0, st>>>(o.locus, inst_of, n, nb, bcnt, flags); note_launch();
  scan_rows<uint32_t>(bcnt, bcnt, nbt, 1, part, bcnt + nbt, st);
  k_bucket_scatter_b<<<nblk(n), 256, 0, st>>>(o.locus, inst_of, n, nb, bcnt, bfill, keys, flags); note_launch();
  k_bucket_sort_keys<<<nblk(nbt, SORT_BUCKETS), SORT_THREADS, 0, st>>>(bcnt, uint32_t(nbt), n, keys, sorted.locus, order, flags);
  k_gather_records<<<nblk(n), 256, 0, st>>>(o.rec, order, n, genome, sorted, inst_sorted, n_inst, nb, bcnt, flags);
  note_launch(2);
}

}  // namespace pg
