"""Edges of the calibration kernel's segments: replicates without sites or of a
few, sizes off the four-site grid, more segments than fit the GPU at a time,
and the Adam steps of one launch against steps taken by hand."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _batch(counts, seed, K=4, J=3):
    """Tables of the given numbers of sites, the replicates of one synthetic
    set cut short."""
    from process_gb300 import calib
    d = calib.synthetic(len(counts), max(max(counts), 1), 80, seed=seed, K=K, J=J)
    idx = np.concatenate([np.arange(int(d.site_off[r]), int(d.site_off[r]) + n) for r, n in enumerate(counts)])
    off = np.r_[0, np.cumsum(counts)].astype(np.uint64)
    cut = calib.CalibData(off, d.alt[idx], d.depth[idx], d.cls[idx], d.signatures, d.epoch_weight, d.phi, d.true_params)
    return calib.batch_of(cut), cut


@pytest.mark.parametrize("counts", [[0, 1, 2, 3], [5, 0, 1023, 1024, 1025, 0], [1027, 4099, 16383, 16389],
                                    [7] * 1300, [40_003, 1, 33_333]])
def test_segments_against_fp64(gpu_lib, counts):
    import torch

    import oracle.calib as oc
    b, d = _batch(counts, seed=3)
    p = torch.tensor(d.true_params + 0.2, dtype=torch.float32, device="cuda")
    nll, grad = b.nll_grad(p)
    again = b.nll_grad(p)
    assert torch.equal(nll, again[0]) and torch.equal(grad, again[1])
    p32 = p.double().cpu().numpy()
    for r in sorted({0, 1, 2, 3, len(counts) - 1} & set(range(len(counts)))):
        n1, g1 = b.nll_grad_one(r, p)
        assert torch.equal(n1[r], nll[r]) and torch.equal(g1[r], grad[r])
        s, e = int(d.site_off[r]), int(d.site_off[r + 1])
        if s == e:
            assert float(nll[r]) == 0.0 and not grad[r].any()
            continue
        f, g = oc.nll_grad(p32[r], d.alt[s:e], d.depth[s:e], d.cls[s:e], d.signatures, d.epoch_weight[r], d.phi[r], 4, 3)
        assert abs(float(nll[r]) - f) / abs(f) < 1e-5
        assert np.linalg.norm(grad[r].double().cpu().numpy() - g) / np.linalg.norm(g) < 1e-4


@pytest.mark.parametrize("counts", [[3000, 0, 1, 2049], [50_001], [900] * 700])
@pytest.mark.parametrize("steps", [1, 2, 6])
def test_adam_steps(gpu_lib, counts, steps):
    """The handle's Adam steps against the same steps on nll_grad's gradients
    in torch (FP32): the updates agree to the rounding of a few operations,
    2e-5 after six steps of 0.05."""
    import torch
    b, d = _batch(counts, seed=4)
    p0 = torch.tensor(d.true_params + 0.3, dtype=torch.float32, device="cuda")
    p = p0.clone()
    nll = b.adam(p, steps, lr=0.05)
    q = p0.clone()
    m, v = torch.zeros_like(q), torch.zeros_like(q)
    for t in range(1, steps + 1):
        f, g = b.nll_grad(q)
        m = 0.9 * m + 0.1 * g
        v = 0.999 * v + 0.001 * g * g
        q = q - 0.05 * (m / (1 - 0.9 ** t)) / (torch.sqrt(v / (1 - 0.999 ** t)) + 1e-8)
    keep = torch.tensor([n >= 900 for n in counts], device="cuda")   # fewer sites: gradients near zero
    assert torch.allclose(p[keep], q[keep], rtol=0, atol=2e-5)
    assert torch.allclose(nll[keep], f[keep], rtol=1e-5)
    empty = torch.tensor([n == 0 for n in counts], device="cuda")
    assert torch.equal(p[empty], p0[empty])
    # a second call starts over
    p2 = p0.clone()
    b.adam(p2, steps, lr=0.05)
    assert torch.equal(p2, p)
