"""Adam steps whose waits run out: the call's results are NaN, the handle reports
it once, and its later calls are right."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_rep,n_sites", [(1, 300), (3, 40_001), (20, 50_000)])
def test_wait_that_runs_out(gpu_lib, n_rep, n_sites):
    import torch

    from process_gb300 import ProcessError, calib
    d = calib.synthetic(n_rep, n_sites, np.linspace(40, 120, n_rep), seed=n_rep)
    b = calib.batch_of(d)
    p0 = torch.tensor(d.true_params + 0.3, dtype=torch.float32, device="cuda")
    want, want_grad = p0.clone(), b.nll_grad(p0)
    want_nll = b.adam(want, 9)
    b.check()
    # no look at all: every wait runs out
    b.L.pg_calib_set_wait_polls(b._h, 0)
    p = p0.clone()
    nll = b.adam(p, 9)
    torch.cuda.synchronize()
    assert torch.isnan(p).all() and torch.isnan(nll).all()
    with pytest.raises(ProcessError, match="ran out"):
        b.check()
    b.check()                                # reported once
    b.L.pg_calib_set_wait_polls(b._h, 2**32 - 1)
    grad = b.nll_grad(p0)
    p = p0.clone()
    nll = b.adam(p, 9)
    b.check()
    assert torch.equal(p, want) and torch.equal(nll, want_nll)
    assert all(torch.equal(x, y) for x, y in zip(grad, want_grad))
