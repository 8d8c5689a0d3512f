"""Wherever the FP32 samplers (pg_fast.cuh) decide a draw, it is the FP64
samplers' draw: 3.1e7 draws in each range of parameters, up to the largest
counts and means a call can have."""
import subprocess
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu

RANGES = {"binomial_halves_small", "binomial_halves", "binomial_halves_large", "binomial_ratios", "binomial_ratios_large",
          "binomial_inversion", "binomial_at_ten", "binomial_rejection", "binomial_masses", "poisson_tiny",
          "poisson_inversion", "poisson_at_ten", "poisson_rejection", "poisson_large"}
# Draws left to the FP64 sampler (they cost time, not results): a band of 2e-4
# around a mean of ten, 1 % of the ranges around it (and every half of 20);
# elsewhere a few in a thousand.
UNDECIDED = 0.03


def test_fp32_draws_are_the_fp64_draws(gpu_lib, tmp_path):
    from process_gb300 import build
    exe = tmp_path / "samplers"
    src = Path(__file__).with_name("samplers.cu")
    subprocess.run([build.nvcc(), *build._flags(False), str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=300)
    print(r.stdout)
    assert r.returncode == 0, r.stdout + r.stderr
    rows = {x[0]: [int(v) for v in x[1:]] for x in map(str.split, r.stdout.splitlines())}
    assert set(rows) == RANGES
    for name, (draws, undecided, wrong) in rows.items():
        assert draws == 608 * 128 * 400
        assert wrong == 0, f"{name}: {wrong} of {draws}"
        assert undecided <= UNDECIDED * draws, f"{name}: {undecided / draws:.2g}"
