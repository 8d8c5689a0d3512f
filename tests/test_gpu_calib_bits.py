"""A replicate's results depend on its sites, their place on the grid of four
and its parameters alone: the same bits in any batch and on either form of the
evaluation (all CTAs resident, or in turn), and 200 Adam steps end where they
always ended."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# parameters after 200 steps of 0.05 from the truth + 0.5 (one replicate of
# 50,000 sites, depth 30 + 1.7 seed); where Adam oscillates it amplifies a
# change of the gradient's rounding to more than the tolerance
AFTER_200 = {
    78: [0.928895831, 0.753292143, 1.11344707, 0.322402388, -0.256808907, -0.834618926, -0.745866776,
         -0.527636409, -1.39237797, -0.205281779, -0.669615388, -0.177816972, -1.44856989, 0.0769839287,
         -3.54400682, -0.871024191, 2.31515503],
    19: [0.343182534, 0.423783392, 1.15212798, 1.07016635, -0.316878051, -0.66213727, -0.912806332,
         -0.677913487, -0.892123044, -0.318275809, -0.263910949, -0.239276215, -2.37355757, -3.20046377,
         0.418218523, -1.72282982, 1.59641302],
    39: [0.394571245, 1.02882385, 0.188571975, 0.55102551, -0.877369523, -0.582913518, -0.374750286,
         -0.0970837548, -0.517373204, -1.8995645, -0.156098112, -1.08724022, -0.698441863, -0.111169584,
         -1.03884292, -0.895890355, 0.42982325],
}


@pytest.mark.parametrize("seed", sorted(AFTER_200))
def test_adam_ends_where_it_did(gpu_lib, seed):
    import torch

    from process_gb300 import calib
    d = calib.synthetic(1, 50_000, 30 + 1.7 * seed, seed=seed)
    b = calib.batch_of(d)
    p = torch.tensor(d.true_params + 0.5, dtype=torch.float32, device="cuda")
    b.adam(p, 200)
    got, want = p.double().cpu().numpy()[0], np.array(AFTER_200[seed])
    assert np.linalg.norm(got - want) / np.linalg.norm(want) < 2e-5


@pytest.mark.parametrize("K,J", [(4, 3), (1, 1), (3, 5), (2, 8), (5, 2), (8, 8)])
def test_same_bits_in_any_batch(gpu_lib, K, J):
    """Replicates of a few sites to several chunks, alone and among enough
    others that the CTAs are not resident together: gradients and Adam steps of
    every shape class of the kernel."""
    import torch

    from process_gb300 import calib
    counts = [40_003, 5, 16_384, 0, 16_385, 2_049]
    rest = 700
    d = calib.synthetic(len(counts), max(counts) + 600, 90, seed=K * 8 + J, K=K, J=J)
    assert all(int(d.site_off[r + 1] - d.site_off[r]) >= n for r, n in enumerate(counts))

    def batch(reps, n):
        idx = np.concatenate([np.arange(int(d.site_off[r]), int(d.site_off[r]) + k) for r, k in zip(reps, n)]).astype(np.int64)
        off = np.r_[0, np.cumsum(n)].astype(np.uint64)
        cut = calib.CalibData(off, d.alt[idx], d.depth[idx], d.cls[idx], d.signatures, d.epoch_weight[reps],
                              d.phi[reps], d.true_params[reps])
        return calib.batch_of(cut), torch.tensor(d.true_params[reps] + 0.3, dtype=torch.float32, device="cuda")

    def results(reps, n):
        b, p = batch(reps, n)
        nll, grad = b.nll_grad(p)
        q = p.clone()
        last = b.adam(q, 12)
        return [x.cpu() for x in (nll, grad, q, last)]

    many = results(list(range(len(counts))) + [5] * rest, counts + [counts[5]] * rest)
    for r in range(len(counts)):
        lead = sum(counts[:r]) % 4               # sites before it, for the same place on the grid
        for x, y in zip(results([0, r], [lead, counts[r]]), many):
            assert torch.equal(x[1], y[r])
