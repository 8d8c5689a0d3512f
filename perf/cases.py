"""Timed cases of the placement, sequencing, batch and calibration paths.

A case is one call (or the few calls that belong together) of a program that
uses this package, through its public entry points:

* ``place``    MutationEngine.place_mutations and the placed table;
* ``seq``      sequence_counts on a placed forest and its counts: the whole
               alt/depth tables or, with ``observed``, the rows with an alt read;
* ``step``     both in a row, the full-scale workload's step;
* ``simulate`` place_mutations and simulate_seq with its result data frame;
* ``genome``   a new MutationEngine (synthesis or upload of the genome, both
               site indices), then one placement from those indices;
* ``batch``    Batch.run over many forests and every instance's counts;
* ``calib``    CalibBatch.nll_grad, one evaluation for all replicates;
* ``adam``     CalibBatch.adam, a calibration loop on the device.

The workloads are those of ``process_gb300.synth``, at other sizes and options.
A case fixes the forest, the rates, the chromosome lengths and the placement
seed, and with them how many mutations are placed; the seed makes the genome's
bases, the signatures and the reads.  Results whose number of rows depends on
the reads go into buffers of the largest size, as a program's own arrays.
Placement and sequencing results are integers and reproducible from their
seeds, so they have no rounding to compare; ``exact`` covers the calibration.
"""
from __future__ import annotations

import math
from dataclasses import replace

import numpy as np
import torch

from process_gb300 import (BasicIlluminaSequencer, ErrorlessIlluminaSequencer, GenomeSpec, sequence_counts,
                           simulate_seq, synth)
from process_gb300 import calib as cal

# sequencing options as synth's workloads set them
FULL_SEQ = dict(coverage=100.0, read_size=150, insert_mean=350, insert_sd=10, insert_model="binomial",
                error_rate=1e-3, purity=0.7, normal=True)
PLAIN_SEQ = dict(coverage=80.0, read_size=150, insert_mean=350, insert_sd=30, insert_model="normal",
                 error_rate=1e-3, purity=1.0, normal=False)


def listed():
    return [
        # a first experiment: 3 x 1 Mbp, 2.5k leaves; the call's latency
        dict(name="place_3mbp", kind="place", workload="plain", leaves=2500),
        # a small chromosome's worth with CNAs, a WGD branch and three epochs
        dict(name="place_155mbp_cna", kind="place", workload="full", scale=0.05, leaves=10000, cna=True),
        # the plain workload's sequencing: 80x paired, discretised normal inserts
        dict(name="seq_3mbp_80x", kind="seq", workload="plain", leaves=2500, observed=False, **PLAIN_SEQ),
        # simulate_seq's own defaults: 10x single-end, error-free, with the normal sample
        dict(name="seq_31mbp_defaults", kind="seq", workload="full", scale=0.01, leaves=1000, cna=False,
             observed=False, coverage=10.0, read_size=150, insert_mean=0, insert_sd=10, insert_model="binomial",
             error_rate=0.0, purity=1.0, normal=True),
        # 100x paired over a genome with CNAs, the usual bulk design
        dict(name="seq_155mbp_cna_100x", kind="seq", workload="full", scale=0.05, leaves=10000, cna=True,
             observed=True, **FULL_SEQ),
        # the full-scale workload: a whole human-sized genome, placed and sequenced
        dict(name="step_3100mbp", kind="step", workload="full", scale=1.0, leaves=10000, cna=True, observed=True,
             **FULL_SEQ),
        # the reference's two calls with the data frame an R user gets
        dict(name="simulate_3mbp", kind="simulate", workload="plain", leaves=2500, **PLAIN_SEQ),
        # a new genome at every position indexed, and a first placement on it
        dict(name="genome_310mbp", kind="genome", workload="full", scale=0.1, leaves=500, cna=False,
             context_sampling=1, uploaded=False),
        # replicates of uneven size on one genome, 30-200x
        dict(name="batch_24x100mbp", kind="batch", n_inst=24, leaves_min=1000, leaves_max=50000,
             genome_len=100_000_000),
        # one table of 2e5 sites: the latency of one gradient
        dict(name="calib_1x2e5", kind="calib", reps=1, sites=200_000, K=4, J=3, depth_min=100.0, depth_max=100.0,
             uneven=False),
        # batched calibration: 512 replicates of 1e5 sites
        dict(name="calib_512x1e5", kind="calib", reps=512, sites=100_000, K=4, J=3, depth_min=30.0,
             depth_max=200.0, uneven=False),
        # a calibration run: 200 Adam steps over 64 replicates
        dict(name="adam_64x5e4", kind="adam", reps=64, sites=50_000, K=4, J=3, depth_min=30.0, depth_max=200.0,
             uneven=False, steps=200),
    ]


def draw(rng):
    def log(lo, hi):
        return math.exp(rng.uniform(math.log(lo), math.log(hi)))

    kind = rng.choice(["place", "seq", "seq", "step", "simulate", "genome", "batch", "calib", "calib", "adam"])
    if kind in ("calib", "adam"):
        c = dict(kind=kind, reps=int(log(1, 512 if kind == "calib" else 64)), sites=int(log(1000, 100_000)) | 1,
                 K=rng.randint(1, 6), J=rng.randint(1, 6), depth_min=rng.uniform(30, 60),
                 depth_max=rng.uniform(60, 200), uneven=rng.random() < 0.5)
        if kind == "adam":         # identifiable parameters: every one has a gradient
            c.update(sites=max(c["sites"], 3001), K=rng.randint(2, 4), J=rng.randint(2, 5), steps=rng.randint(20, 200))
        return c
    if kind == "batch":
        return dict(kind="batch", n_inst=rng.randint(2, 24), leaves_min=100, leaves_max=int(log(1000, 50000)),
                    genome_len=int(log(1_000_000, 100_000_000)))
    c = dict(kind=kind)
    if kind == "simulate" or rng.random() < 0.3:
        c.update(workload="plain", leaves=int(log(30, 10000)))
    else:
        c.update(workload="full", scale=log(0.0005, 0.2), leaves=int(log(30, 10000)), cna=rng.random() < 0.6)
    if kind == "genome":
        c.update(workload="full", scale=log(0.0005, 0.05), leaves=int(log(30, 300)), cna=False,
                 context_sampling=rng.choice([1, 1, 10]), uploaded=rng.random() < 0.5)
    elif kind != "place":
        read = rng.randint(50, 250)
        model = rng.choice(["binomial", "normal"])
        mean = int(read * rng.uniform(1.5, 3.0)) if rng.random() < 0.7 else 0
        sd = rng.randint(1, 12) if model == "binomial" else rng.randint(1, 60)
        if model == "binomial" and mean:
            sd = min(sd, int(math.sqrt(mean) * 0.9))
        c.update(coverage=round(log(5, 200), 1), read_size=read, insert_mean=mean, insert_sd=sd, insert_model=model,
                 error_rate=rng.choice([0.0, 1e-3, 1e-2]), purity=round(rng.uniform(0.2, 1.0), 2),
                 normal=rng.random() < 0.5)
        if kind != "simulate":
            c["observed"] = rng.random() < 0.5
    return c


# ---------------------------------------------------------------- inputs
PLACE_SEED = 7


def _signatures(w, seed):
    """A workload's genome bases and signature vectors made from the seed."""
    rng = np.random.default_rng(seed)
    w.genome = replace(w.genome, seed=seed)
    w.sbs = synth.dirichlet_signatures(rng, len(w.sbs), 96, 0.5, "SBS")
    w.ids = synth.dirichlet_signatures(rng, len(w.ids), 83, 0.5, "ID")


def _workload(case, seed):
    if case["workload"] == "plain":
        w = synth.plain_3mbp(n_leaves=case["leaves"])
        _signatures(w, seed)
        return w
    w = synth.full_scale(n_leaves_per_sample=case["leaves"], genome_scale=case["scale"])
    _signatures(w, seed)
    if not case["cna"]:
        w.mutants = [(name, rates, []) for name, rates, _ in w.mutants]
    if "context_sampling" in case:
        w.context_sampling = case["context_sampling"]
    if case.get("uploaded"):
        # the genome as a program holds it after reading a FASTA file: base
        # codes, with unknown stretches (code 4) at both ends of a chromosome
        rng = np.random.default_rng(seed)
        total = w.genome.total
        bases = rng.integers(0, 4, total, dtype=np.uint8)
        ends = np.cumsum(w.genome.chr_lengths)
        for a, b in zip(np.r_[0, ends[:-1]], ends):
            bases[a:a + (b - a) // 50] = 4
            bases[b - (b - a) // 50:b] = 4
        w.genome = replace(w.genome, bases=bases)
    return w


def _seq_cfg(case):
    return dict(coverage=case["coverage"], read_size=case["read_size"], insert_size_mean=case["insert_mean"],
                insert_size_stddev=case["insert_sd"], insert_model=case["insert_model"],
                error_rate=case["error_rate"], purity=case["purity"], with_normal_sample=case["normal"])


def _place(eng, w):
    return eng.place_mutations(w.forest, w.n_pre_snv, w.n_pre_indel, seed=PLACE_SEED)


def _calib_tables(case, seed):
    """alt, depth and class of every site, drawn from the model on the GPU
    (replicate by replicate of `counts` sites), the model's constants and
    parameters near the truth."""
    R, K, J, C = case["reps"], case["K"], case["J"], 96
    rng = np.random.default_rng(seed)
    counts = (rng.integers(max(1, case["sites"] // 4), case["sites"] + 1, R) if case["uneven"]
              else np.full(R, case["sites"]))
    off = np.r_[0, np.cumsum(counts)].astype(np.uint64)
    sig = rng.dirichlet(np.full(C, 0.5), size=J)
    L = np.tile(np.arange(1, K + 1, dtype=np.float64), (R, 1))
    phi = np.tile(np.array(([1.0, 0.6, 0.35, 0.2] + [0.1] * K)[:K]), (R, 1))
    lr = np.log(rng.uniform(0.5, 2.0, (R, K)))
    w = rng.dirichlet(np.ones(J), size=(R, K))
    purity = rng.uniform(0.5, 0.95, R)
    pi = np.exp(lr) * L
    pi /= pi.sum(axis=1, keepdims=True)
    depth_mean = rng.uniform(case["depth_min"], case["depth_max"], R)
    true = np.concatenate([lr, np.log(np.maximum(w, 1e-3)).reshape(R, K * J),
                           np.log(purity / (1 - purity))[:, None]], axis=1)

    g = torch.Generator(device="cuda").manual_seed(seed)
    dev = dict(device="cuda", dtype=torch.float64)
    rep = torch.repeat_interleave(torch.arange(R, device="cuda"), torch.as_tensor(counts, device="cuda"))
    n = rep.numel()

    def pick(rows, index):     # a category of each row index from cumulative rows
        u = torch.rand(n, generator=g, **dev)
        return (rows.cumsum(1)[index, :-1] < u[:, None]).sum(1)

    k = pick(torch.as_tensor(pi, **dev), rep)
    j = pick(torch.as_tensor(w.reshape(R * K, J), **dev), rep * K + k)
    cdf = torch.as_tensor(sig, **dev).cumsum(1).clamp(max=1.0)
    edges = (cdf + torch.arange(J, **dev)[:, None]).reshape(-1)
    u = j + torch.rand(n, generator=g, **dev)
    cls = (torch.searchsorted(edges, u, right=True) - j * C).clamp(0, C - 1)
    v = torch.as_tensor(purity[:, None] * phi / 2, **dev)[rep, k]
    d = torch.poisson(torch.as_tensor(depth_mean, **dev)[rep].float(), generator=g).clamp(min=1)
    a = torch.binomial(d, v.float(), generator=g)
    host = [x.to(torch.int32).cpu().numpy() for x in (a, d, cls)]
    params = (true + rng.normal(0, 0.3, true.shape)).astype(np.float32)
    return off, *host, sig, L, phi, params


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("calib", "adam"):
        *tables, params = _calib_tables(case, seed)
        return dict(case=case, batch=cal.CalibBatch(*tables), params=torch.as_tensor(params, device="cuda"))
    if kind == "batch":
        w = synth.batch_256(n_inst=case["n_inst"], leaves=(case["leaves_min"], case["leaves_max"]),
                            genome_len=case["genome_len"])
        _signatures(w, seed)
        eng, batch = synth.build_batch(w)
        inst = np.arange(case["n_inst"], dtype=np.uint64)
        return dict(case=case, engine=eng, batch=batch, place_seeds=inst + PLACE_SEED,
                    seq_seeds=inst + np.uint64(1000 * seed))
    w = _workload(case, seed)
    state = dict(case=case, w=w, seed=seed)
    if kind == "genome":
        return state
    state["engine"] = synth.build_engine(w)
    if kind == "place":
        return state
    pf = _place(state["engine"], w)
    M, S = pf.num_of_mutations, len(w.forest.sample_names) + int(case["normal"])
    if kind == "seq":
        state["pf"] = pf
    if kind == "simulate":       # the frame's numeric columns, to be kept by the program
        state["frame"] = {"chr_pos": np.zeros(M, np.int64)}
        for name in w.forest.sample_names + ["normal_sample"][:int(case["normal"])]:
            state["frame"].update({f"{name}.occurrences": np.zeros(M, np.int32),
                                   f"{name}.coverage": np.zeros(M, np.int32), f"{name}.VAF": np.zeros(M)})
    elif case["observed"]:       # page-locked result buffers: row indices, alt, depth
        state["out"] = [torch.zeros(k, dtype=torch.int32, pin_memory=True).numpy() for k in (M, S * M, S * M)]
    return state


# ---------------------------------------------------------------- passes
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "calib":
        return state["batch"].nll_grad(state["params"])
    if kind == "adam":
        params = state["params"].clone()
        nll = state["batch"].adam(params, case["steps"])
        return params, nll
    if kind == "batch":
        batch = state["batch"]
        batch.run(state["place_seeds"], state["seq_seeds"])
        return [batch.counts(i) for i in range(case["n_inst"])]
    w, seed = state["w"], state["seed"]
    if kind == "genome":
        eng = synth.build_engine(w)
        return _ints(eng.index_info()), _ints(_place(eng, w).table())
    pf = state["pf"] if kind == "seq" else _place(state["engine"], w)
    if kind == "place":
        return _ints(pf.table())
    if kind == "simulate":
        rate = case["error_rate"]
        sequencer = BasicIlluminaSequencer(rate) if rate > 0 else ErrorlessIlluminaSequencer()
        cfg = _seq_cfg(case)
        del cfg["error_rate"]
        frame = simulate_seq(pf, sequencer, seed=seed, **cfg)["mutations"]
        for name, col in state["frame"].items():
            col[:len(frame[name])] = frame[name]
        return state["frame"]
    res = sequence_counts(pf, seed, **_seq_cfg(case))
    if not case["observed"]:
        return res.counts()
    index, alt, depth = state["out"]
    rows = len(res.observed(out=(index.view(np.uint32), alt, depth))[0])
    return [rows, *state["out"]]


def _ints(table):
    """A table's 32-bit unsigned columns as the signed view of the same words."""
    return {k: v.view(np.int32) if isinstance(v, np.ndarray) and v.dtype == np.uint32 else v
            for k, v in table.items()}


# ---------------------------------------------------------------- costs
# integer operations of one Philox4x32-10 block with the decisions taken from
# it (a fragment, or one draw of a mutation), and of one read over one locus
DRAW_OPS, VISIT_OPS = 100, 8


def work(case):
    kind = case["kind"]
    if kind in ("calib", "adam"):
        n = case["reps"] * case["sites"] * (0.625 if case["uneven"] else 1.0)
        K, J = case["K"], case["J"]
        flops = n * (K * (4 * J + 14) + 4) * case.get("steps", 1)
        return {"bytes": 12 * n + 8 * case["reps"] * (K + K * J + 2), "flops": flops}
    if kind == "batch":
        # leaves log-uniform, about 2.6 divisions a leaf; SNV rates log-uniform in [1e-8, 1e-7], indels 0.1x
        lo, hi = case["leaves_min"], max(case["leaves_max"], case["leaves_min"] + 1)
        leaves = (hi - lo) / math.log(hi / lo)
        rate = 1.1 * (1e-7 - 1e-8) / math.log(10)
        M = case["n_inst"] * leaves * 2.6 * 2 * case["genome_len"] * rate
        frags = case["n_inst"] * 115 * case["genome_len"] / 300
        return {"bytes": M * (22 + 13 + 8) + case["n_inst"] * leaves * 64,
                "flops": M * 2 * DRAW_OPS + frags * DRAW_OPS + M * 115 * VISIT_OPS}
    w = _workload({**case, "uploaded": False}, 0)
    G = w.genome.total
    rates = w.mutants[0][1]
    div = int(w.forest.divisions.sum())
    M = 2 * G * div * (np.mean(rates["SNV"]) + np.mean(rates["indel"])) + w.n_pre_snv + w.n_pre_indel
    nodes = w.forest.num_of_nodes
    nbytes = flops = 0.0
    if kind != "seq":          # one list entry read and 18 B written per mutation, the forest's columns
        nbytes += M * (4 + 18) + nodes * 32
        flops += M * 2 * DRAW_OPS
    if kind == "genome":       # the bases (2 bits) and the position lists written
        per_id = min(500_000, G)
        nbytes += G / 4 + 4 * G / case["context_sampling"] + 4 * min(83 * per_id, 2 * G)
        nbytes += G if case["uploaded"] else 0
        flops += G * (0 if case["uploaded"] else 25) + G * 8
    if kind in ("seq", "step", "simulate"):
        S = len(w.forest.sample_names) + int(case["normal"])
        frags = S * case["coverage"] * G / (case["read_size"] * (2 if case["insert_mean"] else 1))
        nbytes += M * 13 + S * M * 8
        flops += frags * DRAW_OPS + S * M * case["coverage"] * VISIT_OPS
    return {"bytes": float(nbytes), "flops": float(flops)}


# ---------------------------------------------------------------- 64-bit values
def _nll_grad64(p, a, d, cls, mask, sig, L, phi, K, J):
    """NLL (R) and gradient (R, P) in FP64 over padded tables (R, n)."""
    lr, th, rho = p[:, :K], p[:, K:K + K * J].reshape(-1, K, J), p[:, K + K * J]
    w = torch.softmax(th, dim=2)
    M = w @ sig                                                  # R x K x C
    logw = lr + torch.log(L)
    logpi = logw - torch.logsumexp(logw, dim=1, keepdim=True)    # R x K
    purity = torch.sigmoid(rho)
    v = purity[:, None] * phi / 2
    Mc = torch.stack([torch.gather(M[:, k], 1, cls) for k in range(K)], dim=2)   # R x n x K
    t = (logpi[:, None] + torch.log(Mc) + a[..., None] * torch.log(v)[:, None] +
         (d - a)[..., None] * torch.log1p(-v)[:, None])
    ll = torch.logsumexp(t, dim=2)
    gam = torch.exp(t - ll[..., None]) * mask[..., None]
    G = gam.sum(1)
    grad = torch.empty_like(p)
    grad[:, :K] = -(G - mask.sum(1, keepdim=True) * torch.exp(logpi))
    q = gam / Mc
    for j in range(J):
        H = (q * sig[j][cls][..., None]).sum(1)                  # R x K
        grad[:, K + j:K + K * J:J] = -w[:, :, j] * (H - G)
    A = (gam * a[..., None]).sum(1)
    B = (gam * (d - a)[..., None]).sum(1)
    grad[:, K + K * J] = -(1 - purity) * (A - B * v / (1 - v)).sum(1)
    return -(ll * mask).sum(1), grad


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("calib", "adam"):
        return None            # integers, and ratios of them
    steps = case.get("steps", 1)
    if case["reps"] * case["sites"] * steps > 2_000_000_000:
        return None
    off, a, d, cls, sig, L, phi, params = _calib_tables(case, seed)
    R, K, J = case["reps"], case["K"], case["J"]
    dev = dict(device="cuda", dtype=torch.float64)
    S = torch.as_tensor(sig / sig.sum(axis=1, keepdims=True), **dev)
    off = off.astype(np.int64)
    out = []
    group = max(1, 4_000_000 // case["sites"])
    for r0 in range(0, R, group):
        r1 = min(R, r0 + group)
        n = int((off[r0 + 1:r1 + 1] - off[r0:r1]).max())
        rows = torch.zeros((r1 - r0, n, 3), dtype=torch.int64)
        mask = torch.zeros((r1 - r0, n), dtype=torch.float64)
        for r in range(r0, r1):
            s, e = off[r], off[r + 1]
            for x, col in enumerate((a, d, cls)):
                rows[r - r0, :e - s, x] = torch.from_numpy(col[s:e].astype(np.int64))
            mask[r - r0, :e - s] = 1.0
        rows, mask = rows.cuda(), mask.cuda()
        tab = (rows[..., 0].double(), rows[..., 1].double(), rows[..., 2], mask, S,
               torch.as_tensor(L[r0:r1], **dev), torch.as_tensor(phi[r0:r1], **dev), K, J)
        p = torch.as_tensor(params[r0:r1], **dev)
        if kind == "calib":
            out.append(_nll_grad64(p, *tab))
            continue
        lr, b1, b2, eps = 0.05, 0.9, 0.999, 1e-8
        m, v = torch.zeros_like(p), torch.zeros_like(p)
        for t in range(1, steps + 1):
            nll, g = _nll_grad64(p, *tab)
            m = b1 * m + (1 - b1) * g
            v = b2 * v + (1 - b2) * g * g
            p = p - lr * (m / (1 - b1 ** t)) / (torch.sqrt(v / (1 - b2 ** t)) + eps)
        out.append((p, nll))
    return tuple(torch.cat([o[x] for o in out]) for x in range(2))
