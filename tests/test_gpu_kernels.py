"""Edges of the kernels' dispatch rules and tables, bit-exact against the
oracle's replay: local instance ids and option tables of the read kernel,
insert-size guides, tile windows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _forest_species(o, f):
    return np.array([o.species[(m, ep)] for m, ep in zip(f.mutant, f.epistate)], dtype=np.uint32)


def _copies(kind):
    """Driver lists of the two mutants: few copies (every tile within the read
    kernel's local ids), many (tiles above them), a boundary every few kbp
    (tiles of several parts, then of more parts than the tables hold)."""
    from process_gb300 import CNA, WGD
    if kind == "few":
        return [WGD], [CNA("D", "1", 20_001, 10_000, allele=0), CNA("A", "2", 5_001, 20_000)]
    if kind == "many":
        return [WGD, CNA("A", "1", 10_001, 30_000)], [WGD, CNA("A", "3", 1, 60_000, src_allele=1)]
    return ([CNA("A", "1", 1_001 + 4_000 * i, 2_000) for i in range(14)],
            [CNA("D", "2", 501 + 700 * i, 350, allele=0) for i in range(60)])


READS = [
    # insert tables: a narrow one (several thresholds in most cells of the
    # guide), a wide one, one wider than the guide covers
    dict(coverage=30, read_size=100, insert_size_mean=300, insert_size_stddev=1, insert_model="normal"),
    dict(coverage=15, read_size=75, insert_size_mean=400, insert_size_stddev=60, insert_model="normal"),
    dict(coverage=10, read_size=51, insert_size_mean=3000, insert_size_stddev=500, insert_model="normal"),
    dict(coverage=40, read_size=150, insert_size_mean=0),
]


@pytest.mark.parametrize("copies", ["few", "many", "boundaries"])
@pytest.mark.parametrize("reads", range(len(READS)))
def test_read_kernel_tables(gpu_lib, orc, copies, reads):
    from process_gb300 import synth
    from process_gb300.engine import seq_cfg, sequence_counts
    w = synth.plain_3mbp(seed=11, n_leaves=60)
    w.genome.chr_lengths = [60_000, 60_001, 60_500]
    a, b = _copies(copies)
    (na, ra, _), (nb, rb, _) = w.mutants
    rate = {"SNV": 2e-5, "indel": 4e-6}
    w.mutants = [(na, rate, a), (nb, rate, b)]
    eng = synth.build_engine(w)
    o = orc.OracleEngine.like(w)
    f = w.forest
    pf = eng.place_mutations(f, 60, 6, seed=3)
    op = o.place(f, _forest_species(o, f), 60, 0, 6, 0, seed=3)
    np.testing.assert_array_equal(pf.table()["locus"], op.table()["locus"])
    # the smallest tile; windows with few and with many records; a window
    # longer than the start buckets cover
    for tile in (64, 1000, 9_984, 20_000):
        cfg = dict(error_rate=2e-2, purity=0.6, tile_size=tile, **READS[reads])
        alt, dep = sequence_counts(pf, 17, **cfg).counts()
        c, _ = seq_cfg(chr_index=eng._chr_index, **cfg)
        oalt, odep, _ = op.sequence(c, 17, flavour=0)
        np.testing.assert_array_equal(dep, odep)
        np.testing.assert_array_equal(alt, oalt)


@pytest.mark.parametrize("tile", [64, 448, 8_192])
@pytest.mark.parametrize("coverage", [0.05, 3, 700])
@pytest.mark.parametrize("cna", [False, True])
def test_tile_split(gpu_lib, orc, tile, coverage, cna):
    """Pair counts per tile over chromosomes of one start position, one tile,
    a tile and a bit, one block of 64 tiles more or less, and many: from
    counts in the inversion range of the binomial to large ones, by start
    positions and by DNA mass."""
    from process_gb300 import CNA, synth
    from process_gb300.engine import seq_cfg, sequence_counts
    w = synth.plain_3mbp(seed=5, n_leaves=30)
    w.genome.chr_names = [str(i + 1) for i in range(6)]
    w.genome.chr_lengths = [50, 49 + 64, 49 + 65, 49 + 64 * 64, 49 + 64 * 64 + 1, 40_000]
    (na, ra, _), (nb, rb, _) = w.mutants
    rate = {"SNV": 1e-5, "indel": 1e-6}
    drivers = [CNA("A", "6", 3_001, 7_000), CNA("D", "6", 20_001, 9_000, allele=0)] if cna else []
    w.mutants = [(na, rate, drivers), (nb, rate, [])]
    eng = synth.build_engine(w)
    o = orc.OracleEngine.like(w)
    f = w.forest
    pf = eng.place_mutations(f, 30, 3, seed=2)
    op = o.place(f, _forest_species(o, f), 30, 0, 3, 0, seed=2)
    cfg = dict(coverage=coverage, read_size=50, insert_size_mean=0, error_rate=0.0, purity=0.5, tile_size=tile)
    for seed in (4, 5):
        alt, dep = sequence_counts(pf, seed, **cfg).counts()
        c, _ = seq_cfg(chr_index=eng._chr_index, **cfg)
        oalt, odep, _ = op.sequence(c, seed, flavour=0)
        np.testing.assert_array_equal(dep, odep)
        np.testing.assert_array_equal(alt, oalt)


@pytest.mark.parametrize("infinite", [True, False])
@pytest.mark.parametrize("rate,leaves,sampling", [(1e-6, 8, 1), (6e-5, 40, 1), (2e-4, 60, 1), (2e-5, 60, 10)])
def test_redraws(gpu_lib, orc, infinite, rate, leaves, sampling):
    """Placements from almost no collisions to position lists so full that
    slots take many attempts (and another class from the fourth on), with
    regions that some or all cells have lost on both alleles."""
    from process_gb300 import CNA, SNV, synth
    w = synth.plain_3mbp(seed=8, n_leaves=leaves)
    w.genome.chr_lengths = [40_000, 1_500, 30_011]
    w.context_sampling = sampling
    (na, _, _), (nb, _, _) = w.mutants
    rates = {"SNV": rate, "indel": 0.05 * rate}
    w.mutants = [(na, rates, [SNV("1", 500, "T"), CNA("D", "1", 10_001, 9_000, allele=0),
                              CNA("D", "1", 10_001, 9_000, allele=0)]),
                 (nb, rates, [CNA("D", "3", 1, 20_000, allele=1), CNA("D", "3", 1, 8_000, allele=0)])]
    eng = synth.build_engine(w)
    eng.infinite_sites_model = infinite
    o = orc.OracleEngine.like(w)
    o.set_infinite_sites(infinite)
    f = w.forest
    for seed in (3, 4, 5):
        t = eng.place_mutations(f, 40, 5, seed=seed).table()
        ot = o.place(f, _forest_species(o, f), 40, 0, 5, 0, seed=seed).table()
        assert len(t["locus"]) == len(ot["locus"])
        for k in ("locus", "edge", "aux", "cls", "sig", "allele", "kind", "nature"):
            np.testing.assert_array_equal(t[k], ot[k], err_msg=k)


@pytest.mark.parametrize("rate", [1e-9, 1e-4, 1e-3, 4e-3])
def test_edge_counts(gpu_lib, orc, rate):
    """Mutations per (edge, epoch): Poisson means in the inversion range, near
    its end and far above it; edges that start or end at an epoch's start or
    span epochs."""
    from process_gb300 import SamplesForest, synth
    w = synth.plain_3mbp(seed=9, n_leaves=50)
    w.genome.chr_lengths = [3_000, 3_000, 3_000]
    f0 = w.forest
    nodes = f0.get_nodes()
    birth = np.round(f0.birth_time)                       # many edges end exactly at an epoch's start
    w.forest = SamplesForest(nodes["cell_id"], nodes["ancestor"], np.full(f0.num_of_nodes, "A", dtype=object),
                             np.full(f0.num_of_nodes, "", dtype=object), nodes["sample"], birth,
                             np.arange(f0.num_of_nodes) % 7 + 1)
    w.mutants = [("A", {"SNV": [rate, 2 * rate, 0.5 * rate], "indel": [0.1 * rate, 0.0, rate]}, [])]
    t_end = float(birth.max())
    w.exposures = [(t, {"SBS1": 1.0, "ID1": 1.0}) for t in (0.0, np.round(t_end / 3), np.round(t_end / 2))]
    eng = synth.build_engine(w)
    eng.infinite_sites_model = False
    o = orc.OracleEngine.like(w)
    o.set_infinite_sites(False)
    f = w.forest
    sp = np.zeros(f.num_of_nodes, dtype=np.uint32)
    for seed in (1, 2):
        t = eng.place_mutations(f, 3, 2, seed=seed).table()
        ot = o.place(f, sp, 3, 0, 2, 0, seed=seed).table()
        np.testing.assert_array_equal(t["edge"], ot["edge"])
        np.testing.assert_array_equal(t["locus"], ot["locus"])


@pytest.mark.parametrize("sampling,max_rep", [(1, 1), (1, 40), (2, 1000), (7, 500_000), (1023, 3), (1024, 100), (5000, 17)])
def test_index_strides(gpu_lib, orc, sampling, max_rep):
    """Position lists at strides from 1 to beyond a round of the emit pass,
    over repeats, chromosomes that start and end inside a round, and unknown
    stretches."""
    from process_gb300 import GenomeSpec, MutationEngine
    rng = np.random.default_rng(sampling)
    lengths = [9_001, 31, 4_097, 1, 20_000]
    bases = rng.integers(0, 4, sum(lengths)).astype(np.uint8)
    bases[500:900] = 2                                     # long runs and short repeats
    bases[5_000:6_000] = np.tile([0, 3], 500)
    bases[12_000:14_000] = np.resize([1, 0, 2, 2, 3], 2_000)
    bases[3_000:3_100] = 4
    bases[13_100] = 4
    g = GenomeSpec(["a", "b", "c", "d", "e"], lengths, bases=bases)
    eng = MutationEngine(g, context_sampling=sampling, max_repetition_storage=max_rep)
    o = orc.OracleEngine(lengths, bases, context_sampling=sampling, max_rep=max_rep)
    for which, n in ((0, 32), (1, 83)):
        for k in range(n):
            np.testing.assert_array_equal(eng.read_index(which, k), o.read_index(which, k), err_msg=f"{which} {k}")


@pytest.mark.parametrize("reads", [0, 3])
@pytest.mark.parametrize("tile", [64, 192, 448, 1_088, 2_304, 2_560, 10_048])
def test_read_windows_by_records(gpu_lib, orc, tile, reads):
    """Windows of a few records to more than shared memory holds (0.05 per
    position): every number of lanes that share a record, tiles in one atom
    and across atoms, one and several batches of fragments."""
    from process_gb300 import CNA, synth
    from process_gb300.engine import seq_cfg, sequence_counts
    w = synth.plain_3mbp(seed=12, n_leaves=50)
    w.genome.chr_lengths = [30_000, 900, 20_011]
    (na, _, _), (nb, _, _) = w.mutants
    rate = {"SNV": 5e-5, "indel": 2e-6}
    w.mutants = [(na, rate, [CNA("A", "1", 8_001, 12_000)]), (nb, rate, [CNA("D", "3", 1, 9_000, allele=1)])]
    eng = synth.build_engine(w)
    o = orc.OracleEngine.like(w)
    f = w.forest
    pf = eng.place_mutations(f, 2_000, 50, seed=6)
    op = o.place(f, _forest_species(o, f), 2_000, 0, 50, 0, seed=6)
    cfg = dict(error_rate=5e-3, purity=0.7, with_normal_sample=True, tile_size=tile, **READS[reads])
    alt, dep = sequence_counts(pf, 23, **cfg).counts()
    c, _ = seq_cfg(chr_index=eng._chr_index, **cfg)
    oalt, odep, _ = op.sequence(c, 23, flavour=0)
    np.testing.assert_array_equal(dep, odep)
    np.testing.assert_array_equal(alt, oalt)


@pytest.mark.parametrize("leaves,epochs", [(3, 1), (682, 3), (683, 3), (2_730, 3), (2_731, 3)])
def test_edge_offsets_by_size(gpu_lib, orc, leaves, epochs):
    """Placements whose (edge, epoch) cells fill less than a chunk of the
    one-launch prefix sum, one chunk, a chunk and a bit, and more than it
    takes."""
    from process_gb300 import synth
    w = synth.plain_3mbp(seed=4, n_leaves=leaves)
    w.genome.chr_lengths = [70_000, 30_001]
    w.genome.chr_names = ["1", "2"]
    first = w.exposures[0][1] if w.exposures else {}
    w.exposures = [(float(t * 10), first) for t in range(epochs)]
    (na, _, _), (nb, _, _) = w.mutants
    rate = {"SNV": 2e-9 * 1000 / leaves, "indel": 1e-9}
    w.mutants = [(na, rate, []), (nb, rate, [])]
    eng = synth.build_engine(w)
    o = orc.OracleEngine.like(w)
    f = w.forest
    pf = eng.place_mutations(f, 500, 20, seed=9)
    op = o.place(f, _forest_species(o, f), 500, 0, 20, 0, seed=9)
    for col in ("locus", "edge", "aux"):
        np.testing.assert_array_equal(pf.table()[col], op.table()[col])


@pytest.mark.parametrize("infinite", [True, False])
def test_no_allele_left(gpu_lib, infinite):
    """A class whose every position the cells have lost on both alleles: the
    call fails, whatever the draws left in the columns, and the engine goes
    on."""
    from process_gb300 import CNA, SBS_CLASSES, DomainError, GenomeSpec, synth
    w = synth.plain_3mbp(seed=3, n_leaves=20)
    bases = np.zeros(60_000, np.uint8)                       # poly-A, and A C A repeats on the second
    bases[40_000:] = np.resize([0, 1], 20_000)
    w.genome = GenomeSpec(["1", "2"], [40_000, 20_000], bases=bases)
    sig = np.zeros(96)
    sig[SBS_CLASSES.index("A[C>T]A")] = 1.0
    w.sbs = {"SBS1": sig}
    (na, _, _), (nb, _, _) = w.mutants
    lost = [CNA("D", "2", 1, 20_000, allele=0), CNA("D", "2", 1, 20_000, allele=0)]
    w.mutants = [(na, {"SNV": 1e-5, "indel": 0.0}, lost), (nb, {"SNV": 1e-5, "indel": 0.0}, [])]
    eng = synth.build_engine(w)
    eng.infinite_sites_model = infinite
    with pytest.raises(DomainError, match="left"):
        eng.place_mutations(w.forest, 0, 0, seed=2)
    ok = synth.plain_3mbp(seed=3, n_leaves=20)
    assert synth.build_engine(ok).place_mutations(ok.forest, 10, 1, seed=2).num_of_mutations > 0
