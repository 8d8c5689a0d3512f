"""Index lists of genomes whose units are shared by 16, 8, ... warps of the emit
pass, on both sides of each size where that number changes (1,824 warps, units
of 4,096 bases)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("units", [1, 113, 114, 115, 228, 229, 456, 457, 912, 913])
@pytest.mark.parametrize("sampling,max_rep", [(1, 500_000), (3, 400)])
def test_lists_by_units(gpu_lib, orc, units, sampling, max_rep):
    from process_gb300 import GenomeSpec, MutationEngine
    rng = np.random.default_rng(units)
    n = 4_096 * units - int(rng.integers(0, 4_000))
    bases = rng.integers(0, 4, n).astype(np.uint8)
    at = rng.integers(0, n - 60, n // 500)
    for i, a in enumerate(at):                             # runs and short repeats
        bases[a:a + 40] = np.resize(bases[a:a + 1 + i % 6], 40)
    bases[n // 2:n // 2 + 30] = 4
    lengths = [n // 3, n - n // 3]
    eng = MutationEngine(GenomeSpec(["1", "2"], lengths, bases=bases), context_sampling=sampling, max_repetition_storage=max_rep)
    o = orc.OracleEngine(lengths, bases, context_sampling=sampling, max_rep=max_rep)
    for which, classes in ((0, 32), (1, 83)):
        for k in range(classes):
            np.testing.assert_array_equal(eng.read_index(which, k), o.read_index(which, k), err_msg=f"{which} {k}")
