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
