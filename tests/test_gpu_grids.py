"""Calls whose blocks do not fit one dimension of a grid."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_batch_of_many_samples(gpu_lib, orc):
    """An instance of 70,001 samples (a grid's second dimension ends at 65,535)
    beside one of two: every sample's reads as the oracle's."""
    from process_gb300 import Batch, MutationEngine, synth
    from process_gb300.engine import seq_cfg
    w = synth.plain_3mbp(seed=6, n_leaves=30)
    w.genome.chr_names, w.genome.chr_lengths = ["1", "2"], [1_500, 701]
    w.context_sampling = 1
    name, rates = w.mutants[0][0], {"SNV": 1e-8, "indel": 0.0}
    w.mutants = [(name, rates, [])]
    expo = np.zeros(len(w.sbs))
    expo[0] = 1.0
    w.exposures = [(0.0, {list(w.sbs)[0]: 1.0, list(w.ids)[0]: 1.0})]
    forests = [synth.birth_forest(70_001, 70_001, 3, subclone=None, mutant=name),
               synth.birth_forest(40, 2, 4, subclone=None, mutant=name)]
    cfg = dict(coverage=12.0, read_size=100, insert_size_mean=0, error_rate=1e-3, purity=0.5, tile_size=512)
    eng = MutationEngine(w.genome, w.sbs, w.ids, context_sampling=1)
    b = Batch(eng, forests, [rates["SNV"]] * 2, [0.0] * 2, np.tile(expo, (2, 1)),
              np.tile(np.eye(len(w.ids))[0], (2, 1)), [cfg] * 2, n_pre_snv=[25, 25], n_pre_indel=[0, 0])
    b.tile_sizes = [512, 512]
    b.run([5, 6], [7, 8])
    for i, f in enumerate(forests):
        w.forest = f
        o = orc.OracleEngine.like(w)
        sp = np.array([o.species[(m, e)] for m, e in zip(f.mutant, f.epistate)], dtype=np.uint32)
        op = o.place(f, sp, 25, 0, 0, 0, seed=5 + i)
        c, _ = seq_cfg(chr_index=eng._chr_index, **cfg)
        oalt, odep, _ = op.sequence(c, 7 + i, flavour=0)
        alt, dep = b.counts(i)
        assert alt.shape == oalt.shape == ((70_002 if i == 0 else 3), b.dims(i)[0])      # and the normal sample
        np.testing.assert_array_equal(dep, odep)
        np.testing.assert_array_equal(alt, oalt)


@pytest.mark.parametrize("cna", [False, True])
def test_tile_split_of_many_samples_and_chromosomes(gpu_lib, orc, cna):
    """600 samples of 60,001 chromosomes, one of them far longer than the others:
    the tile split has more blocks (62 for each sample and chromosome) than a
    grid (2^31 - 1)."""
    from process_gb300 import CNA, synth
    from process_gb300.engine import seq_cfg, sequence_counts
    w = synth.plain_3mbp(seed=5, n_leaves=30)
    n, samples = 60_000, 600
    w.genome.chr_names = [str(i) for i in range(n + 1)]
    w.genome.chr_lengths = [60] * n + [1_000_000]
    name = w.mutants[0][0]
    w.mutants = [(name, {"SNV": 1e-9, "indel": 0.0}, [CNA("A", str(n), 300_001, 400_000)] if cna else [])]
    f = w.forest = synth.birth_forest(samples, samples, 3, subclone=None, mutant=name)
    eng = synth.build_engine(w)
    o = orc.OracleEngine.like(w)
    sp = np.array([o.species[(m, e)] for m, e in zip(f.mutant, f.epistate)], dtype=np.uint32)
    pf = eng.place_mutations(f, 200, 0, seed=2)
    op = o.place(f, sp, 200, 0, 0, 0, seed=2)
    cfg = dict(coverage=0.5, read_size=50, insert_size_mean=0, error_rate=0.0, purity=0.5, tile_size=64)
    alt, dep = sequence_counts(pf, 4, **cfg).counts()
    c, _ = seq_cfg(chr_index=eng._chr_index, **cfg)
    oalt, odep, _ = op.sequence(c, 4, flavour=0)
    assert (alt.shape[0] - 1) * (n + 1) * ((1_000_000 - 49) // 64 // 256 + 1) >= 2**31
    np.testing.assert_array_equal(dep, odep)
    np.testing.assert_array_equal(alt, oalt)
