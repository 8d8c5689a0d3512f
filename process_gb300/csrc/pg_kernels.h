// Host-callable launchers of the device kernels and the plain-pointer
// structures they take.  Everything here is internal to the library; the
// public boundary is include/process_gb300.h.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace pg {

// Philox key of a call (the seed's two words)
struct Key { uint32_t k0, k1; };
__host__ __device__ inline Key make_key(uint64_t seed) {
  return {uint32_t(seed), uint32_t(seed >> 32)};
}

constexpr uint32_t MAX_EPOCHS = 16;

// Counts kernel launches of this library (read with pg_launch_count).
void note_launch(uint32_t n = 1);

// ---------------------------------------------------------------- index
void genome_synth(uint32_t* words, uint64_t G, uint64_t seed, double gc, cudaStream_t st);
void genome_pack(uint32_t* words, const uint8_t* codes, uint64_t G, cudaStream_t st);
// unknown bases (codes > 3, e.g. N) as one bit per position ((G + 31) / 32
// words); *any (zeroed by the caller) becomes 1 when there is one.  A NULL
// mask below means a genome without unknown bases.
void genome_nmask(const uint8_t* codes, uint64_t G, uint32_t* mask, uint32_t* any, cudaStream_t st);
uint32_t index_num_tiles(uint64_t G);
// bases at pos (BASE_INVALID for positions outside the genome or unknown)
void genome_gather(const uint32_t* g, const uint32_t* nmask, uint64_t G, const uint32_t* pos, uint64_t n,
                   uint8_t* out, cudaStream_t st);
// per placed mutation rows[i] (all rows when NULL): {locus, ref code, alt
// code, kind | signature << 8 | nature << 16}; the codes hold up to 8
// characters of "ACGNT" coded 1..5, 4 bits each, the first character highest
void row_info(const uint32_t* locus, const uint32_t* aux, const uint8_t* kind, const uint8_t* sig,
              const uint8_t* nature, const uint32_t* rows, uint64_t n, const uint32_t* g, const uint32_t* nmask,
              uint64_t G, uint4* out, cudaStream_t st);
int index_num_classes(int which);  // 0 = SBS contexts (32), 1 = ID classes (83)
// allocation-free per-class totals over a caller-held genome (see pg_index.cu);
// returns nullptr on success, else a message
constexpr uint32_t NOALLOC_MAX_TILES = 8192;
const char* index_counts_noalloc(int which, const uint32_t* g, uint64_t G, const uint32_t* chr_off, int n_chr,
                                 uint64_t* totals, cudaStream_t st);
// contexts and repeat sites that touch an unknown base are not indexed; the
// SBS contexts (which 0) also skip the positions set in amask (regions to
// avoid; NULL: none)
void index_count(int which, const uint32_t* g, const uint32_t* nmask, const uint32_t* amask, uint64_t G,
                 const uint32_t* chr_off, int n_chr, uint32_t* cnt, uint32_t* part, uint32_t* totals, cudaStream_t st);
void genome_avoid_mask(const uint32_t* pos, uint64_t n, uint32_t* mask, cudaStream_t st);
// every: all strides are 1 (each indexed position is written)
void index_emit(int which, const uint32_t* g, const uint32_t* nmask, const uint32_t* amask, uint64_t G,
                const uint32_t* chr_off, int n_chr, const uint32_t* cnt_scanned, const uint32_t* stride,
                const uint64_t* list_off, const uint32_t* list_len, uint32_t* lists, bool every, cudaStream_t st);

// ---------------------------------------------------------------- genome classes
// Copy-number events are rare, so the cells of a forest fall into few
// genotype classes: the genome below each CNA/WGD event edge.  A class is a
// list of segments (absolute [start, end), ascending) with the sorted ids of
// the allele instances covering each segment.  Class 0 is the germline:
// instances 0 and 1 over every chromosome.
struct GenomeClasses {
  uint32_t n_classes;
  const uint32_t* node_class;   // class of each edge's genome after its own events (n_nodes + 1 entries)
  const uint32_t* seg_off;      // n_classes + 1
  const uint32_t* seg_start;
  const uint32_t* seg_end;
  const uint32_t* seg_ioff;     // covering instances: inst_list[seg_ioff, seg_ioff + seg_icnt)
  const uint32_t* seg_icnt;
  const uint16_t* inst_list;
};

// ---------------------------------------------------------------- placement
struct PlaceTables {
  // forest (device)
  uint32_t n_nodes;
  const int32_t* parent;
  const double* birth;
  const uint32_t* species;
  const uint32_t* divisions;
  // epochs and rates (device); rates are [species][epoch]
  uint32_t n_epochs;
  const double* epoch_start;
  const double* snv_rate;
  const double* indel_rate;
  const double* cna_rate;       // per species (passenger CNAs per base per division)
  const double* node_size;      // allelic size of each edge's genome (n_nodes + 1 entries)
  GenomeClasses gc;
  // signatures: exposure CDFs [(n_epochs+1) rows][n_sigs], class CDFs [n_sigs][classes]
  uint32_t n_sbs_sigs, n_id_sigs;
  const uint32_t* sbs_expo_cdf;
  const uint32_t* sbs_sig_cdf;
  const uint32_t* id_expo_cdf;
  const uint32_t* id_sig_cdf;
  // indices
  const uint32_t* genome;
  const uint64_t* ctx_off; const uint32_t* ctx_len; const uint32_t* ctx_lists;
  const uint64_t* id_off; const uint32_t* id_len; const uint32_t* id_lists;
};

// SoA of placed mutations (device)
struct PlaceOut {
  uint32_t* locus;    // absolute position (SNV) or anchor position (indel)
  uint32_t* edge;     // node index; n_nodes = preneoplastic edge
  uint32_t* aux;      // SNV: alt base; indel: descriptor
  uint8_t* cls;       // SBS96 / ID83 class, 0xff for drivers
  uint8_t* sig;       // signature index (cause), 0xff for drivers
  uint16_t* allele;   // allele instance
  uint16_t* seq;      // order on the edge: driver event index, 0x7fff passengers, 0 preneoplastic
  uint8_t* kind;
  uint8_t* nature;
};

// Mutations in slot order, before the sort: the locus and a record {edge, aux,
// allele | seq << 16, cls | sig << 8 | kind << 16 | nature << 24}
struct PlaceRaw {
  uint32_t* locus;
  uint4* rec;
};

struct DriverRec {
  uint32_t locus, edge, aux, allele, seq;   // allele: the instance, chosen on the host
  uint8_t kind, pad[3];
};

void place_cna_counts(const PlaceTables& t, uint32_t* cnt_cna, uint64_t seed, double germline_size, cudaStream_t st);
void place_edge_counts(const PlaceTables& t, uint32_t* cnt_snv, uint32_t* cnt_id, uint64_t seed,
                       uint32_t n_pre_snv, uint32_t n_pre_id, cudaStream_t st);
void place_drivers(const PlaceRaw& o, const DriverRec* drv, uint32_t n_drv, uint32_t base_slot, cudaStream_t st);
// the first draw of slots [0, n_slots); with first, fused with their insertion
// into the first round's table `first` (fmask + 1 entries, all ones on entry;
// lost: n_slots bytes of scratch).  Then sites_first_finish inserts the
// drivers' loci and lists the losing slots in next.
void place_first_round(const PlaceTables& t, const PlaceRaw& o, uint64_t seed, const uint32_t* off_snv,
                       const uint32_t* off_id, uint32_t n_snv, uint32_t n_slots, unsigned long long* first,
                       uint32_t fmask, uint8_t* lost, uint32_t* err, cudaStream_t st);
void sites_first_finish(const uint32_t* drv_locus, uint32_t n_drv, unsigned long long* first, uint32_t fmask,
                        uint8_t* lost, uint32_t n_slots, uint32_t* next, uint32_t* n_next, uint32_t* err,
                        cudaStream_t st);
// The redraws of the *n (<= n_max, in device memory) slots of list: keys and
// held (both all ones) have cap entries, a power of two >= 2 n_max.  ctl
// (zeroed) reports the rounds (one more than the last attempt needed; 0:
// nothing was pending) and the status.
constexpr uint32_t TAIL_MAX_ROUND = 256;
enum : uint32_t { TAIL_ROUNDS_EXHAUSTED = 1u };
struct TailCtl {
  uint32_t status;
  uint32_t rounds;
};
void sites_settle(const PlaceTables& t, const PlaceRaw& o, uint64_t seed, const uint32_t* off_snv,
                  const uint32_t* off_id, uint32_t n_snv, const uint32_t* list, const uint32_t* n, uint32_t n_max,
                  const unsigned long long* first, uint32_t fmask, uint32_t* keys, unsigned long long* held,
                  uint64_t cap, TailCtl* ctl, uint32_t* err, cudaStream_t st);
// without infinite sites: redraws of the slots whose locus has no allele
void sites_covered(const PlaceTables& t, const PlaceRaw& o, uint64_t seed, const uint32_t* off_snv,
                   const uint32_t* off_id, uint32_t n_snv, uint32_t n_slots, TailCtl* ctl, uint32_t* err,
                   cudaStream_t st);
// What says that a placement failed (tail may be NULL): a sort then writes nothing.
struct PlaceFlags {
  const uint32_t* err;
  const TailCtl* tail;
};
uint32_t sort_num_buckets(uint64_t G);
// sort by (locus, slot) into `sorted`; bcnt: 2 sort_num_buckets(G) entries,
// keys: n 64-bit keys
void sort_by_locus(const PlaceRaw& o, uint32_t n, const uint32_t* genome, uint64_t G, uint32_t* bcnt, uint32_t* part,
                   uint32_t* order, const PlaceOut& sorted, unsigned long long* keys, const PlaceFlags& flags,
                   cudaStream_t st);

// ---------------------------------------------------------------- sequencing
struct SeqRec {            // 16 B, one per placed mutation, sorted by locus
  uint32_t locus;
  uint32_t tin, tout;      // Euler interval of the edge that carries it
  uint32_t info;           // instance | (order on the edge & 0x7fff) << 16 | kind << 31
};

// fragments the read kernel handles per shared-memory batch (5 per thread);
// tiles are sized so that their fragment count rarely exceeds one batch
constexpr uint32_t SEQ_FRAGS_PER_BATCH = 1280;

// The insert-size lookup of a 31-bit word v: entry g = v >> 21 of the guide
// covers the words of one cell and holds k, the first index whose threshold
// exceeds the cell's first word (bits 0-9), whether words past that threshold
// need a walk over the following ones (bit 10; else they get k + 1), and the
// last word of the cell that still gets k, relative to the cell's first (bits
// 11-31: one comparison with the word's own low bits at the top).  Tables
// of at most SEQ_GUIDE_INS thresholds have a guide: 1024 cells leave about
// one word in a hundred of a normal-shaped table to the walk (256 left one in
// thirty, so that most warps had a lane in it).
constexpr uint32_t SEQ_GUIDE = 1024, SEQ_GUIDE_INS = 1024;
// Cells are asked for in ascending order: at is the previous cell's entry (0
// at the first).
inline uint32_t insert_guide(const uint32_t* thr, uint32_t n, uint32_t g, uint32_t& at) {
  const uint32_t first = g << 21, next = first + (1u << 21);   // cells end at 2^31 at the latest
  while (at < n && thr[at] <= first) ++at;
  const uint32_t lo = at;
  if (lo >= n || thr[lo] >= next) return (lo < n ? lo : n - 1) | 0xfffff800u;
  const bool walk = lo + 1 >= n || thr[lo + 1] < next;
  return lo | (thr[lo] - first - 1u) << 11 | (walk ? 0x400u : 0u);
}

struct SeqTiles {
  uint32_t n_tiles;        // over all selected chromosomes
  uint32_t* start;   // first start position of the tile (absolute)
  uint32_t* len;     // number of start positions in the tile
  uint32_t* chr_end; // absolute end of the tile's chromosome
  uint32_t* rec_lo;  // records of the tile's window [start, start + len - 1 + span)
  uint32_t* rec_hi;
};

struct SeqSample {
  uint32_t n_leaves;
  uint32_t leaf_off;       // into leaf_tin
  uint32_t normal_thr;     // read from a normal cell iff u < normal_thr
  uint32_t all_normal;     // the normal sample: every read from a normal cell
  // with copy-number events: the sample's cell options (option 0 its normal
  // cells, then the genotype classes of its leaves, ascending) and, per atom,
  // the thresholds of the option draw (rows of n_opt at opt_cdf_off)
  uint32_t opt_off, n_opt, opt_cdf_off;
};

// The thresholds that split a substitution error's word range [0, thr) into
// the three other bases: [0, t1), [t1, t2), [t2, thr).
inline void err_thirds(uint32_t thr, uint32_t& t1, uint32_t& t2) {
  t1 = thr / 3u;
  t2 = uint32_t(uint64_t(thr) * 2u / 3u);
}

struct SeqParams {
  uint32_t read_len;
  uint32_t paired;
  uint32_t span;           // max fragment span past the start (read_len or max insert)
  uint32_t ins_min, n_ins; // insert size = ins_min + index in the CDF table
  const uint32_t* ins_cdf;
  const uint32_t* ins_guide; // SEQ_GUIDE entries (see insert_guide), 16-byte aligned
  uint32_t err_thr;        // substitution error iff u < err_thr
  uint32_t err_t1, err_t2; // the erroneous base: the first of the three others iff u < err_t1,
                           //   the second iff err_t1 <= u < err_t2, else the third
  uint32_t normal_tin;     // Euler index of normal cells
  uint32_t n_alleles;
  // copy-number state (has_cna == 0: every cell has instances 0 and 1 everywhere)
  uint32_t has_cna;
  GenomeClasses gc;
  const uint32_t* chain_off;  // instance lineage: for instance y, ancestors chain_anc[chain_off[y]..]
  const uint16_t* chain_anc;  //   with the order key (tin << 16 | seq + 1) of the copy that led towards y
  const uint64_t* chain_key;
  // Atoms: the coarsest partition of the genome into intervals on which every
  // class's covering instances are constant.  A tile's start range is cut
  // into parts, one per atom it meets.
  uint32_t n_classes;         // row length of atom_ioff / atom_icnt
  const uint32_t* atom_ioff;  // [atom * n_classes + class]: first covering instance in gc.inst_list
  const uint32_t* atom_icnt;  //   and their number (0: the class has no allele there)
  const uint32_t* part_off;   // parts of tile t: [part_off[t], part_off[t + 1])
  const uint32_t* part_start; // absolute first start position of the part
  const uint32_t* part_len;
  const uint32_t* part_atom;
  const uint32_t* part_cdf;   // [sample * n_parts + part]: thresholds of the part draw within its tile
  uint32_t n_parts;
  const uint32_t* opt_class;  // per cell option: genotype class
  const uint32_t* opt_leaf_off;   // its leaves in cls_leaf_tin
  const uint32_t* opt_nleaf;      // 0: the normal cells
  const uint32_t* cls_leaf_tin;   // every sample's leaves grouped by class (Euler indices)
  const uint32_t* opt_cdf;        // option thresholds (see SeqSample)
  // for a tile inside one atom: the atom (else 0xffffffff), and the draw
  // tables of (sample, atom), row sample * n_atoms + atom (see CnRow)
  const uint32_t* tile_atom;
  const struct CnRow* cn_rows;
  uint32_t n_atoms;
  const uint32_t* nmask;          // unknown reference bases (N), one bit each, or NULL (SAM output)
};

// The chromosomes of a sequencing call: tile t of slot c (first[c] <= t <
// first[c] + ntiles[c], k = t - first[c]) covers the starts
// [start[c] + k T, + min(T, nstarts[c] - k T)).
struct SeqChroms {
  uint32_t n_slots;
  const uint32_t *first, *ntiles, *start, *nstarts, *end;
  const uint32_t* depth;    // levels of the tile-split tree
  const uint32_t* id;       // chromosome numbers (keys of the tree's draws)
  const uint64_t* pairs;    // fragments
  uint32_t T, n_tiles, max_tiles;
};
// What the read kernel needs that depends on no copy-number table, in one
// launch: the tiles and the ranges of their windows' records, the records
// and, for the first n_split samples (all, or none), the fragments per tile
// by start positions (see seq_tile_counts).
void seq_prepare(const SeqChroms& c, const SeqTiles& tiles, const PlaceOut& sorted, uint32_t n_recs,
                 const uint32_t* edge_tin, const uint32_t* edge_tout, uint32_t span, SeqRec* recs, uint32_t n_split,
                 uint64_t seed, uint32_t* pair_cnt, cudaStream_t st);
// Copy-number tables of a sequencing call.  Parts: tile t's start range cut
// at atom boundaries, at part_off[t] .. part_off[t + 1] (part_off holds
// n_tiles + 1 entries; `part` is scan scratch of scan_part_elems(n_tiles, 1)).
void seq_tile_parts(uint32_t n_tiles, const uint32_t* tile_start, const uint32_t* tile_len,
                    const uint32_t* atom_start, uint32_t n_atoms, uint32_t genome_len, uint32_t* part_off,
                    uint32_t* scan_part, uint32_t* part_start, uint32_t* part_len, uint32_t* part_atom,
                    uint32_t* tile_atom,
                    cudaStream_t st);
// Per (sample, tile) its integer copy sums (I0, S) (scratch tile_sums,
// 2 * n_samples * n_tiles) and, for tiles of several parts, the thresholds
// of the part draw (part_cdf[s * n_parts + part]); then per (sample,
// chromosome slot) the mass before each tile (mass_cum[s * n_tiles + t]) and
// the slot's total (mass_tot[s * n_slots + slot]), each the mass of the
// exact integer sums before it.  A stretch with integer copy sums (I0, S)
// weighs wn * I0 + (wt / nl) * S (the second term when nl > 0);
// icnt0 / copy_sum are per (sample, atom).
void seq_tile_mass(uint32_t n_samples, uint32_t n_slots, const uint32_t* c_first, const uint32_t* c_ntiles,
                   const uint32_t* part_off, const uint32_t* part_len, const uint32_t* part_atom, uint32_t n_atoms,
                   const double* wn, const double* wt, const uint64_t* nl, const uint64_t* icnt0,
                   const uint64_t* copy_sum, uint32_t n_tiles, uint32_t n_parts, uint64_t* tile_sums,
                   double* mass_cum, double* mass_tot, uint32_t* part_cdf, cudaStream_t st);
// ---------------------------------------------------------------- SAM records
// One aligned read as the SAM writer needs it; the host formats the text.
constexpr uint32_t SAM_MAX_CIGAR = 16;
struct SamRead {
  uint32_t pos;             // absolute first aligned reference position
  uint32_t mate_pos;        // absolute first position of the mate (paired reads)
  int32_t tlen;             // signed template length (0 for single-end reads)
  uint16_t flag;            // SAM FLAG
  uint16_t n_cigar;
  uint32_t seq_len;
  uint32_t cigar[SAM_MAX_CIGAR];   // op length << 4 | op (0 M, 1 I, 2 D)
};
// Reads of tiles [t0, t0 + n_chunk) (global tile indices, for the draws) of
// every sample: the fragment draws of the read kernel, each mate's bases
// built from the genome with the mutations its allele instance carries and
// the substitution errors of its error words.  Read r of the fragment j of
// (sample s, tile t0 + k) is written at 2 * (out_off[s * n_chunk + k] + j) +
// mate (one slot per fragment for single-end reads); seq holds max_len
// bytes per read.
void seq_sam_reads(const SeqRec* recs, uint32_t n_recs, const uint32_t* aux, const uint32_t* genome,
                   const SeqTiles& tiles, uint32_t t0, uint32_t n_chunk, const uint32_t* pair_cnt,
                   const SeqSample* samples, uint32_t n_samples, const uint32_t* leaf_tin, const SeqParams& prm,
                   uint64_t seed, const uint64_t* out_off, SamRead* out, char* seq, uint32_t max_len,
                   cudaStream_t st);

// The copy-number draw tables of one (atom, sample), laid out for a read CTA:
// per cell option its threshold (the last one takes what is left; unused ones
// past any 31-bit word), its covering instances, leaves, first leaf and the
// mate tag of its first instance.  The instances of all options are numbered
// through as local ids (the instance of id l: linst[l]); n_ids exceeds
// SEQ_CN_IDS when they, or the options, do not fit (the row is then not used).
constexpr uint32_t SEQ_CN_OPTS = 8, SEQ_CN_IDS = 16;
struct alignas(16) CnRow {
  uint32_t thr[SEQ_CN_OPTS];
  uint4 opt[SEQ_CN_OPTS];
  uint32_t linst[SEQ_CN_IDS];
  uint32_t n_ids, pad[3];
};

// ---------------------------------------------------------------- batched sequencing
// Per-instance descriptor of a batch: every table row below is relative to the
// instance's offsets, so each instance computes exactly what the plain path
// computes for it alone with the same tile size and seed.
struct SeqInst {
  SeqParams prm;
  uint32_t n_samples, sample_off;   // rows of the batch's SeqSample array
  uint32_t n_tiles, tile_off;       // rows of the batch's tile arrays
  uint32_t T;                       // tile size
  uint32_t slot_off;                // chromosome tables
  uint32_t n_blocks, blk_off;       // tile-split blocks of 64 tiles (a warp each)
  uint32_t etin_off;                // edge Euler table rows (n_nodes + 2)
  uint64_t pair_off;                // pair counts [sample][tile]
  uint64_t count_off;               // alt/depth of sample s: count_off + s * count_stride + record
  uint32_t count_stride;            // >= the instance's mutations
};
struct SeqBatch {
  uint32_t n_inst;
  const SeqInst* inst;
  const Key* keys;                  // sequencing key of each instance
  const uint32_t* rec_off;          // n_inst + 1: records of instance i (filled by placement)
  const uint32_t* cnt_off;          // n_inst + 1: first tile-split warp of each instance
  uint32_t max_samples, n_cnt, n_tiles_all;
  const uint32_t *tile_start, *tile_len, *tile_end, *tile_inst;
  uint32_t *rec_lo, *rec_hi;        // per tile, relative to the instance's first record
  const uint32_t *c_first, *c_ntiles, *c_depth, *c_nstarts, *c_id;
  const uint64_t* c_pairs;
  const uint32_t *blk_slot, *blk_index;
  uint32_t* pair_cnt;
  const SeqSample* samples;
  const uint32_t* leaf_tin;
  const uint32_t *etin, *etout;
  uint32_t *alt, *depth;
};
// batched placement (launchers in pg_place.cu): cells of instance i are
// [cell_off[i], cell_off[i+1]); node_off counts each instance's nodes plus its
// preneoplastic edge
void place_edge_counts_batch(const PlaceTables* tabs, uint32_t n_inst, const uint32_t* node_off, uint32_t n_nodes_all,
                             const uint32_t* cell_off, const Key* keys, const uint32_t* pre_snv, const uint32_t* pre_id,
                             uint32_t* cnt_snv, uint32_t* cnt_id, cudaStream_t st);
// the first draw of a batch's slots; with fkeys (fmask + 1 entries, all ones)
// also the first infinite-sites round (fslot: as many entries, all ones;
// lost: n_slots bytes), whose losers go to next
void place_first_round_batch(const PlaceTables* tabs, uint32_t n_inst, const uint32_t* cell_off, const Key* keys,
                             const PlaceRaw& o, uint16_t* inst_of, const uint32_t* off_snv, const uint32_t* off_id,
                             uint32_t n_snv, uint32_t n_slots, uint64_t* fkeys, uint32_t* fslot, uint64_t fmask,
                             uint8_t* lost, uint32_t* next, uint32_t* n_next, uint32_t* err, cudaStream_t st);
// sites_settle for a batch, keyed by (instance << 32 | locus)
void sites_settle_batch(const PlaceTables* tabs, uint32_t n_inst, const uint32_t* cell_off, const Key* keys,
                        const PlaceRaw& o, uint16_t* inst_of, const uint32_t* off_snv, const uint32_t* off_id,
                        uint32_t n_snv, const uint32_t* list, const uint32_t* n, uint32_t n_max, const uint64_t* fkeys,
                        uint64_t fmask, uint64_t* hkeys, unsigned long long* held, uint64_t cap, TailCtl* ctl,
                        uint32_t* err, cudaStream_t st);
// sort by (instance, locus, slot); bcnt holds n_inst * sort_num_buckets(G)
// + 1 entries and ends as the exclusive scan of the bucket counts; keys: n
// 64-bit keys
void sort_batch(const PlaceRaw& o, const uint16_t* inst_of, uint32_t n, uint32_t n_inst, const uint32_t* genome,
                uint64_t G, uint32_t* bcnt, uint32_t* bfill, uint32_t* part, uint32_t* order, const PlaceOut& sorted, uint16_t* inst_sorted,
                unsigned long long* keys, const PlaceFlags& flags, cudaStream_t st);
// records of the first *n_dev sorted mutations of a batch (cap >= *n_dev)
void seq_batch_records(const PlaceOut& sorted, const uint16_t* inst_sorted, const uint32_t* n_dev, uint32_t cap,
                       const SeqBatch& b, SeqRec* recs, cudaStream_t st);
// tile split, record ranges and the read kernel over every (tile, sample)
void seq_batch_reads(const SeqBatch& b, const SeqRec* recs, cudaStream_t st);
// per (sample, tile) pair counts: multinomial split of each chromosome's
// pair count over its tiles by a binary tree of binomial draws.  Tiles weigh
// their number of start positions (seq_prepare), or their DNA mass:
// mass_cum[s * n_tiles + t] is the sample's mass of the chromosome's tiles
// before t and mass_tot[s * n_slots + slot] the chromosome's total.
void seq_tile_counts(const SeqChroms& c, uint32_t n_samples, const double* mass_cum, const double* mass_tot,
                     uint64_t seed, uint32_t* pair_cnt, cudaStream_t st);
// observed rows: flag[m] = 1 when some sample has an alt read of mutation m;
// with pos the exclusive scan of the flags (n_active rows), the compact
// [sample][row] alt / depth tables and each row's mutation index
void seq_active_flags(const uint32_t* alt, uint32_t n_samples, uint64_t M, uint32_t* flag, cudaStream_t st);
void seq_active_gather(const uint32_t* alt, const uint32_t* depth, uint32_t n_samples, uint64_t M, const uint32_t* pos,
                       uint32_t n_active, uint32_t* index, uint32_t* a_out, uint32_t* d_out, cudaStream_t st);
// the rows prm.cn_rows of n_samples samples (prm's other copy-number fields set)
void seq_cn_rows(const SeqParams& prm, const SeqSample* samples, uint32_t n_samples, CnRow* rows, cudaStream_t st);
void seq_reads(const SeqRec* recs, uint32_t n_recs, const SeqTiles& tiles, const uint32_t* pair_cnt,
               const SeqSample* samples, uint32_t n_samples, const uint32_t* leaf_tin, const SeqParams& prm,
               uint64_t seed, uint32_t* alt, uint32_t* depth, cudaStream_t st);

// ---------------------------------------------------------------- calibration
struct CalibArgs {
  uint32_t K, J, C, P;          // epochs, signatures, classes, parameters per replicate
  const int32_t* alt;           // sites of all replicates, concatenated (16-byte aligned columns)
  const int32_t* depth;
  const int32_t* cls;
  const uint64_t* site_off;     // n_rep + 1
  const float* epoch_w;         // n_rep x K  (L_k: relative length of epoch k)
  const float* phi;             // n_rep x K  (mean cellular fraction of epoch-k mutations)
  const float* sig_rows;        // C x JP: S_j(c) by class, JP = 4 (J <= 4) or 8 floats, zero beyond J
  // A replicate's chunks of CAL_CHUNK sites (chunk c: those from
  // site_off + c CAL_CHUNK on) and segments, the CTAs it is dealt out to: a
  // chunk each, or with by_warps the chunks' warps in turn (a replicate without
  // sites has one segment)
  const uint32_t* rep_first_chunk;  // n_rep + 1
  const uint32_t* rep_first_seg;    // n_rep + 1
  const uint32_t* seg_rep;
  uint32_t by_warps;
  uint32_t* rep_done;             // n_rep counts, zero before a launch of one evaluation (and after it), all ones
                                  //   before one of several
  float* partial;                 // per chunk, or per warp of a chunk, part_stride sums (>= 1 + 3K + K J): n_rows rows,
  uint32_t part_stride, n_rows;   //   with steps > 1 twice that
  uint32_t seg0, rep0;            // first segment and replicate of the launch
  uint32_t steps;                 // evaluations of the launch (above 1: Adam steps, without tab)
  uint32_t* rep_left;             // several evaluations: n_rep words, all ones before the launch, 0 where a CTA left
  uint32_t wait_polls;            //   a wait after this many looks, which
  uint32_t* status;               //   sets this
  float* tab;                     // per replicate, calib_tab floats: its constants, where they and the
                                  //   epilogues have launches of their own; else NULL
};
struct AdamArgs {               // m == nullptr: no optimizer step
  float* m; float* v;
  uint32_t t;                   // the step's number, from 0 (launches of one step)
  float lr, beta1, beta2, eps;
};
// one evaluation over the segments [a.seg0, a.seg0 + n_segs): whole replicates
void calib_launch(const CalibArgs& a, uint32_t n_segs, uint32_t n_rep, float* params, float* nll, float* grad,
                  const AdamArgs& adam, cudaStream_t st);
int calib_ctas_per_sm(uint32_t K, uint32_t J);   // resident CTAs of the evaluation kernel
uint32_t calib_chunk();                          // sites of a chunk
uint32_t calib_tab(uint32_t K, uint32_t J);      // floats of a replicate in CalibArgs::tab

}  // namespace pg
