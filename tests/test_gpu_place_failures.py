"""Placements that find no room: the call fails in good time, however many of its
mutations are left over, and the engine goes on."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_pre", [4_000, 300_000, 2_000_000])
def test_more_mutations_than_loci(gpu_lib, n_pre):
    """Infinite sites on 3,000 bases, every position indexed: all but 3,000 of
    the mutations are given up (a thread would take hours to sort two million
    of them in one bucket)."""
    import time

    from process_gb300 import DomainError, synth
    w = synth.plain_3mbp(seed=3, n_leaves=20)
    w.genome.chr_lengths = [1_000, 1_000, 1_000]
    w.context_sampling = 1
    w.mutants = [(name, {"SNV": 0.0, "indel": 0.0}, []) for name, _, _ in w.mutants]
    eng = synth.build_engine(w)
    t0 = time.perf_counter()
    with pytest.raises(DomainError, match="no free locus"):
        eng.place_mutations(w.forest, n_pre, 0, seed=2)
    assert time.perf_counter() - t0 < 20
    assert eng.place_mutations(w.forest, 30, 3, seed=2).num_of_mutations == 33


def test_batch_with_more_mutations_than_loci(gpu_lib):
    from process_gb300 import Batch, DomainError, GenomeSpec, MutationEngine, synth
    rng = np.random.default_rng(1)
    eng = MutationEngine(GenomeSpec(["1"], [3_000], seed=4), synth.dirichlet_signatures(rng, 1, 96, 0.5, "SBS"),
                         synth.dirichlet_signatures(rng, 1, 83, 0.5, "ID"), context_sampling=1)
    forests = [synth.birth_forest(20, 1, seed, subclone=None, mutant="A") for seed in (1, 2, 3)]
    cfgs = [dict(coverage=5.0, read_size=50, insert_size_mean=0)] * 3
    one = np.ones((3, 1))
    b = Batch(eng, forests, [0.0] * 3, [0.0] * 3, one, one, cfgs, n_pre_snv=[10, 200_000, 10], n_pre_indel=[0, 0, 0])
    with pytest.raises(DomainError, match="no free locus"):
        b.run(np.arange(3), np.arange(3))
    b = Batch(eng, forests, [0.0] * 3, [0.0] * 3, one, one, cfgs, n_pre_snv=[10, 20, 10], n_pre_indel=[0, 0, 0])
    b.run(np.arange(3), np.arange(3))
    assert [b.dims(i)[0] for i in range(3)] == [10, 20, 10]
