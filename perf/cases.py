"""Timed cases of the tree-scoring paths: what a phylogenetics program has the
library do, through the package's public calls.

Every case draws its own tree, model and alignment from the seed.  Tip
states are evolved down the tree on the GPU (each branch redraws a site with
a probability set by its length and the site's rate), so neighbouring tips
share states as real alignments do; a few per cent of the cells are
ambiguous or missing.  A program that searches trees calls these entry
points with a different tree each time, and so do the passes here: states of
different seeds hold different trees on one context.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from phylocaml_gb300 import _native, batch, costmatrix, fitch, likelihood, likelihood_c, mlmodel, mlp, spr, tree

DEV = "cuda:0"


def listed():
    return [
        # parsimony score of a genome-scale DNA alignment: the node sets and
        # step counts of one candidate tree (4-bit state sets)
        {"name": "fitch_dna_large", "kind": "fitch", "tips": 1024, "sites": 1000000, "lanes": 4},
        # one gene in the 8-bit layout, rescored for every candidate tree of a
        # search: a call of a few microseconds
        {"name": "fitch_bv8_small", "kind": "fitch", "tips": 64, "sites": 1337, "lanes": 8},
        # step-matrix parsimony of DNA under an integerised model, tabulated
        {"name": "tcm_dna", "kind": "tcm", "tips": 512, "sites": 250001, "states": 4, "rule": "general"},
        # step-matrix parsimony of amino acids (medians formed from the matrix)
        {"name": "tcm_protein", "kind": "tcm", "tips": 128, "sites": 20003, "states": 20, "rule": "metric"},
        # lnL of a concatenated alignment, float pairs, codes kept on the device
        {"name": "prune_pair_large", "kind": "prune", "tips": 512, "patterns": 446427, "rates": 4,
         "precision": 48},
        # lnL of one small gene from host arrays in the default precision
        {"name": "prune_host_small", "kind": "prune_host", "tips": 32, "patterns": 1000, "rates": 4,
         "precision": 32},
        # one gradient of a maximum-likelihood model fit: 2 x 9 + 1 models of
        # one tree (central differences over GTR + Gamma4 + frequencies)
        {"name": "fit_models", "kind": "fit", "tips": 64, "patterns": 15159, "rates": 4, "models": 19,
         "precision": 48},
        # the node-by-node likelihood operator folded over a tree, nodes reused
        {"name": "fold_nodes", "kind": "fold", "tips": 128, "patterns": 100003, "rates": 4, "precision": 32},
        # many gene families at once: protein and codon models on their own trees
        {"name": "batch_mixed", "kind": "batch", "variants": 32, "tips": 128, "min_patterns": 5000,
         "max_patterns": 100000},
        # every SPR neighbour of a new tree scored exactly
        {"name": "spr_scan", "kind": "scan", "tips": 128, "patterns": 16852, "rates": 4, "precision": 48},
        # one round of a learned SPR search but for its network: branch
        # lengths re-estimated, the features of every move, the top 32 scored
        {"name": "spr_round", "kind": "round", "tips": 256, "patterns": 45675, "rates": 4, "precision": 48,
         "moves": 32},
        # that round's network: every move ranked, then eight training steps
        {"name": "mlp_rank_train", "kind": "mlp", "rows": 257048, "batch": 1024, "steps": 8},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fitch", "fitch", "tcm4", "tcm", "prune", "prune_host", "fit", "fold", "batch", "scan",
                       "round", "mlp"])
    if kind == "fitch":
        lanes = rng.choice([4, 4, 8, 8, 16, 32, 64])
        tips = _log(rng, 16, 1024)
        return {"kind": kind, "tips": tips, "sites": _log(rng, 300, min(1e6, 4e9 / (lanes * tips))),
                "lanes": lanes}
    if kind == "tcm4":
        return {"kind": "tcm", "tips": _log(rng, 16, 512), "sites": _log(rng, 300, 250000), "states": 4,
                "rule": rng.choice(["general", "metric"])}
    if kind == "tcm":
        return {"kind": kind, "tips": _log(rng, 8, 128), "sites": _log(rng, 300, 20000),
                "states": rng.choice([5, 8, 12, 20, 22]), "rule": rng.choice(["general", "metric"])}
    if kind == "prune":
        return {"kind": kind, "tips": _log(rng, 16, 512), "patterns": _log(rng, 1000, 440000),
                "rates": rng.choice([1, 4, 4, 4]), "precision": rng.choice([32, 48, 48, 48])}
    if kind == "prune_host":
        return {"kind": kind, "tips": _log(rng, 8, 128), "patterns": _log(rng, 100, 20000),
                "rates": rng.choice([1, 2, 4, 4]), "precision": rng.choice([32, 48, 64])}
    if kind == "fit":
        return {"kind": kind, "tips": _log(rng, 16, 64), "patterns": _log(rng, 1000, 15000), "rates": 4,
                "models": rng.randint(3, 19), "precision": 48}
    if kind == "fold":
        return {"kind": kind, "tips": _log(rng, 8, 128), "patterns": _log(rng, 500, 50000),
                "rates": rng.choice([1, 4, 4]), "precision": rng.choice([32, 64])}
    if kind == "batch":
        lo = _log(rng, 500, 5000)
        return {"kind": kind, "variants": rng.randint(2, 32), "tips": _log(rng, 16, 128), "min_patterns": lo,
                "max_patterns": _log(rng, lo, 60000)}
    if kind == "scan":
        return {"kind": kind, "tips": _log(rng, 12, 128), "patterns": _log(rng, 500, 16000), "rates": 4,
                "precision": rng.choice([32, 48, 48])}
    if kind == "round":
        return {"kind": kind, "tips": _log(rng, 16, 200), "patterns": _log(rng, 1000, 40000), "rates": 4,
                "precision": 48, "moves": rng.choice([32, 256])}
    return {"kind": "mlp", "rows": _log(rng, 2000, 250000), "batch": rng.choice([512, 1000, 1024]), "steps": 8}


# ---- inputs -------------------------------------------------------------------

def _evolve(tr, states, sites, gen, rates=None):
    """Tip states [tips, sites] (uint8) on the GPU: along a branch each site is
    redrawn uniformly with probability 1 - exp(-rate t S / (S - 1))."""
    out = torch.empty((tr.n_tips, sites), dtype=torch.uint8, device=DEV)
    live = {tr.n_nodes - 1: torch.randint(0, states, (sites,), dtype=torch.uint8, device=DEV, generator=gen)}
    k = states / (states - 1.0)
    for v in tr.depth_first_order():
        parent = live.pop(v)
        for c in (int(tr.left[v - tr.n_tips]), int(tr.right[v - tr.n_tips])):
            t = float(tr.brlen[c]) * k
            p = -math.expm1(-t) if rates is None else -torch.expm1(rates * -t)
            hit = torch.rand(sites, device=DEV, generator=gen) < p
            new = torch.randint(0, states, (sites,), dtype=torch.uint8, device=DEV, generator=gen)
            row = torch.where(hit, new, parent)
            if c < tr.n_tips:
                out[c] = row
            else:
                live[c] = row
    return out


def _generators(seed):
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed))
    return np.random.default_rng(int(seed)), gen


def _site_rates(rates, sites, gen):
    r = torch.as_tensor(rates, dtype=torch.float32, device=DEV)
    return r[torch.randint(0, len(rates), (sites,), device=DEV, generator=gen)]


def _dna_codes(tr, sites, gen, rates=None):
    """4-bit DNA masks: 3 % of the cells ambiguous or missing."""
    masks = torch.ones((), dtype=torch.uint8, device=DEV) << _evolve(tr, 4, sites, gen, rates)
    for row in masks:
        u = torch.rand(sites, device=DEV, generator=gen)
        other = torch.randint(0, 4, (sites,), dtype=torch.uint8, device=DEV, generator=gen)
        row |= torch.where(u < 0.015, torch.ones_like(other) << other, torch.zeros_like(other))
        row |= torch.where(u > 0.985, torch.full_like(other, 15), torch.zeros_like(other))
    return masks


def _state_sets(tr, states, sites, gen):
    """Bit-set codes (int64) of an alphabet of any size, 2 % of the cells sets
    of two states and 1 % missing (every state)."""
    codes = torch.empty((tr.n_tips, sites), dtype=torch.int64, device=DEV)
    one = torch.ones((), dtype=torch.int64, device=DEV)
    every = -1 if states == 64 else (1 << states) - 1
    for i, row in enumerate(_evolve(tr, states, sites, gen)):
        u = torch.rand(sites, device=DEV, generator=gen)
        c = one << row.long()
        c |= torch.where(u < 0.02, one << torch.randint(0, states, (sites,), device=DEV, generator=gen),
                         torch.zeros_like(c))
        codes[i] = torch.where(u > 0.99, torch.full_like(c, every), c)
    return codes


def _pack(codes, lanes):
    """Rows of lanes packed into 32-bit words, rows a multiple of 16 bytes."""
    rows, sites = codes.shape
    if lanes == 4:
        codes = codes.to(torch.uint8)
        if sites % 2:
            codes = torch.nn.functional.pad(codes, (0, 1))
        codes = codes[:, 0::2] | (codes[:, 1::2] << 4)
    else:
        codes = codes.to({8: torch.uint8, 16: torch.int16, 32: torch.int32, 64: torch.int64}[lanes])
    codes = codes.contiguous().view(torch.uint8)
    width = codes.shape[1]
    out = torch.zeros((rows, (width + 15) // 16 * 16), dtype=torch.uint8, device=DEV)
    out[:, :width] = codes
    return out.view(torch.int32)


def _gtr(rng, rates):
    """GTR exchangeabilities (the last fixed at 1), frequencies, and rate
    classes (the means of four equal shares of a Gamma(0.5); otherwise drawn)."""
    co = rng.uniform(0.5, 2.0, 5)
    pi = rng.dirichlet([5.0] * 4)
    r = {1: np.ones(1), 4: np.array([0.03338775, 0.25191592, 0.82026848, 2.89442785])}.get(rates)
    if r is None:
        r = np.sort(rng.gamma(1.0, 1.0, rates)) + 0.05
        r = r / r.mean()
    return co, pi, r, np.full(rates, 1.0 / rates)


def _dna_spec(co, pi, rates, probs):
    return mlmodel.Spec(("GTR", list(co)), ("DiscreteCustom", list(zip(rates, probs))),
                        ("Empirical", list(pi)), 4)


def _dna_table():
    t = ((np.arange(16)[:, None] >> np.arange(4)) & 1).astype(np.float64)
    t[0] = 1.0
    return t


def _dna_problem(case, seed):
    """Tree, model parameters, codes [tips, patterns] on the GPU and weights."""
    rng, gen = _generators(seed)
    tr = tree.yule(case["tips"], rng, 0.08)
    par = _gtr(rng, case["rates"])
    n = case["patterns"]
    codes = _dna_codes(tr, n, gen, _site_rates(par[2], n, gen))
    # pattern counts: mostly 1, a tail of common patterns
    w = torch.as_tensor(np.minimum(rng.geometric(0.6, n), 50).astype(np.float64), device=DEV)
    return rng, gen, tr, par, codes, w


def _padded(codes, multiple):
    rows, n = codes.shape
    out = torch.zeros((rows, (n + multiple - 1) // multiple * multiple), dtype=torch.uint8, device=DEV)
    out[:, :n] = codes
    return out


def _fit_models(rng, par, count):
    """The point and its neighbours along the parameters, as a gradient asks."""
    co, pi, rates, probs = par
    out = []
    for i in range(count):
        x = np.concatenate([np.log(co), np.log(pi[:-1] / pi[-1]), [0.0]])
        if i:
            x[(i - 1) // 2 % len(x)] += 1e-4 if i % 2 else -1e-4
        e = np.exp(np.append(x[5:8], 0.0))
        r = rates ** math.exp(x[8])
        out.append((np.exp(x[:5]), e / e.sum(), r / (r * probs).sum(), probs))
    return out


def _variants(case, seed):
    """(tree, q, pi, rates, probs, codes, patterns) of each variant: protein
    models of four rate classes and codon models in turn."""
    rng, gen = _generators(seed)
    out = []
    for k in range(case["variants"]):
        tr = tree.yule(case["tips"], rng, 0.1)
        s = 20 if k % 2 == 0 else 61
        ex = np.triu(rng.lognormal(0.0, 1.0, (s, s)), 1)
        if s == 61:   # most codon changes need more than one step and are rare
            ex *= np.where(rng.random((s, s)) < 0.15, 1.0, 0.01)
        pi = rng.dirichlet(np.full(s, 5.0))
        q = (ex + ex.T) * pi
        np.fill_diagonal(q, -q.sum(1))
        q /= -(np.diag(q) * pi).sum()
        rates, probs = (np.array([0.03338775, 0.25191592, 0.82026848, 2.89442785]), np.full(4, 0.25)) \
            if s == 20 else (np.ones(1), np.ones(1))
        # pattern counts spread evenly over the range, in no order
        n = case["min_patterns"] + int((case["max_patterns"] - case["min_patterns"]) * (0.618034 * (k + 1) % 1.0))
        codes = _evolve(tr, s, n, gen, _site_rates(rates, n, gen))
        gap = torch.rand(codes.shape, device=DEV, generator=gen) < 0.01
        codes = torch.where(gap, torch.full_like(codes, s), codes)
        w = torch.as_tensor(np.minimum(rng.geometric(0.6, n), 50).astype(np.float64), device=DEV)
        out.append((tr, q, pi, rates, probs, codes, w, n))
    return out


def _state_table(s):
    return np.concatenate([np.eye(s), np.ones((1, s))])


def _network(case, seed):
    """He-uniform weights, move features and targets of a ranking network."""
    rng, gen = _generators(seed)
    parts = []
    for rows, cols in ((256, 64), (256, 256), (256, 256), (1, 256)):
        a = math.sqrt(6.0 / cols)
        parts += [rng.uniform(-a, a, rows * cols), np.zeros(rows)]
    params = np.concatenate(parts).astype(np.float32)
    scale = torch.exp(torch.randn(64, device=DEV, generator=gen))
    x = torch.randn((case["rows"], 64), device=DEV, generator=gen) * scale + scale.flip(0)
    t = torch.asinh(-torch.exp(2.0 * torch.randn(case["rows"], device=DEV, generator=gen)) * 10.0)
    return params, x, t


def _tcm(rng, states, rule):
    """Substitution costs: a metric of few distinct costs, or an integerised
    model's (-10^4 log of a transition probability)."""
    if rule == "general":
        return np.trunc(-1e4 * np.log(rng.dirichlet(np.ones(states) * 2, states) * 0.25 + 1e-6)).astype(np.int32)
    c = rng.integers(1, 4, (states, states))
    c = np.minimum(c, c.T)
    np.fill_diagonal(c, 0)
    for k in range(states):
        c = np.minimum(c, c[:, [k]] + c[[k], :])
    return c.astype(np.int32)


def prepare(case, seed):
    kind, ctx = case["kind"], _native.default_context()
    s = {"case": case, "ctx": ctx}
    if kind in ("fitch", "tcm"):
        rng, gen = _generators(seed)
        n = case["sites"]
        s["tree"] = tree.yule(case["tips"], rng, 0.08)
        if kind == "fitch":
            lanes = case["lanes"]
            codes = _dna_codes(s["tree"], n, gen) if lanes <= 8 else \
                _state_sets(s["tree"], {16: 12, 32: 20, 64: 61}[lanes], n, gen)
        else:
            s["matrix"] = costmatrix.CostMatrix(_tcm(rng, case["states"], case["rule"]), case["rule"])
            lanes = s["matrix"].lane_bits()
            codes = _dna_codes(s["tree"], n, gen) if case["states"] == 4 else \
                _state_sets(s["tree"], case["states"], n, gen)
        s["tips"] = _pack(codes, lanes)
        s["lanes"], s["ld"] = lanes, s["tips"].shape[1]
        s["weights"] = torch.randint(1, 9, (n,), dtype=torch.int32, device=DEV, generator=gen)
        s["sets"] = torch.zeros((case["tips"] - 1, s["ld"]), dtype=torch.int32, device=DEV)
        s["cost"] = torch.zeros(n, dtype=torch.int32, device=DEV)
        s["total"] = torch.zeros(1, dtype=torch.int64, device=DEV)
    elif kind == "batch":
        s["batch"] = batch.Batch(
            [batch.Variant(tr, q, pi, r, p, _state_table(len(pi)), _padded(codes, 128), w, n)
             for tr, q, pi, r, p, codes, w, n in _variants(case, seed)], ctx, batch.Options(True, "cost"))
        s["lnl"] = torch.zeros(case["variants"], dtype=torch.float64, device=DEV)
        s["site"] = torch.zeros(s["batch"].patterns, dtype=torch.float64, device=DEV)
    elif kind == "mlp":
        params, x, t = _network(case, seed)
        s["net"] = mlp.MLP(seed=1, max_batch=case["batch"], ctx=ctx)
        s["net"].set_params(params)
        s["net"].fit_norm(x)
        s["x"] = x
        b = case["batch"]
        s["steps"] = [(x[i * b % len(x):][:b].contiguous(), t[i * b % len(x):][:b].contiguous())
                      for i in range(case["steps"])]
    else:
        rng, gen, tr, par, codes, w = _dna_problem(case, seed)
        s["tree"], s["table"] = tr, _dna_table()
        if kind == "fit":
            s["models"] = [mlmodel.create(_dna_spec(*m), ctx, eigen=False)
                           for m in _fit_models(rng, par, case["models"])]
        else:
            s["model"] = mlmodel.create(_dna_spec(*par), ctx)
        if kind in ("prune_host", "fit", "fold"):
            s["codes"], s["weights"] = codes.cpu().numpy(), w.cpu().numpy()
        else:
            s["codes"], s["weights"] = _padded(codes, 16), w
        if kind == "prune":
            s["lnl"] = torch.zeros(1, dtype=torch.float64, device=DEV)
            s["site"] = torch.zeros(case["patterns"], dtype=torch.float64, device=DEV)
        if kind == "fold":
            s["lk"] = likelihood_c.LkModel(s["model"], s["table"], case["patterns"], s["weights"],
                                           case["precision"], ctx)
            s["nodes"] = None
        if kind in ("scan", "round"):
            s["engine"] = spr.SprEngine(s["codes"], case["patterns"], s["model"], s["table"], w,
                                        case["precision"], ctx)
            if kind == "round":
                s["engine"].set_tree(tr)
                s["top"] = np.sort(rng.choice(s["engine"].n_moves, case["moves"], replace=False))
    return s


# ---- one pass -------------------------------------------------------------------

def run(s):
    c, ctx = s["case"], s["ctx"]
    kind = c["kind"]
    if kind == "fitch":
        fitch.fitch_tree_dev(s["tree"], s["tips"], s["ld"], c["sites"], s["lanes"], s["weights"], s["sets"],
                             s["cost"], s["total"], ctx)
        return s["sets"], s["cost"], s["total"]
    if kind == "tcm":
        s["matrix"].tree_cost_dev(s["tree"], s["tips"], s["ld"], c["sites"], s["weights"], s["sets"],
                                  s["cost"], s["total"], ctx)
        return s["sets"], s["cost"], s["total"]
    if kind == "prune":
        likelihood.tree_lnl_dev(s["tree"], s["model"], s["codes"], s["codes"].shape[1], c["patterns"],
                                s["table"], s["weights"], s["lnl"], c["precision"], s["site"], ctx)
        return s["lnl"], s["site"]
    if kind == "prune_host":
        return likelihood.tree_lnl(s["tree"], s["model"], s["codes"], s["table"], s["weights"], c["precision"],
                                   ctx, site_lnl=True)
    if kind == "fit":
        return likelihood.tree_lnl_models(s["tree"], s["models"], s["codes"], s["table"], s["weights"],
                                          c["precision"], ctx)
    if kind == "fold":
        s["nodes"], minus_lnl = likelihood_c.fold_postorder(s["lk"], s["tree"], s["codes"], s["nodes"])
        return minus_lnl, s["nodes"][-1].root_cost(site_lnl=True)[1]
    if kind == "batch":
        s["batch"].run_dev(s["lnl"], s["site"])
        return s["lnl"], s["site"]
    if kind == "scan":
        s["engine"].set_tree(s["tree"])
        return s["engine"].scan()
    if kind == "round":
        e = s["engine"]
        e.set_tree(s["tree"])
        lnl = e.optimize(2, 1e-4)
        return lnl, e.lengths()[0], e.features(), e.score(s["top"])
    pred = s["net"].forward(s["x"])
    for x, t in s["steps"]:
        s["net"].train_step(x, t, None, 2e-3, 1e-4, sync=False)
    return pred, s["net"].params()


# ---- the work a pass cannot do without ------------------------------------------

def work(case):
    kind = case["kind"]
    if kind in ("fitch", "tcm"):
        n, sites = case["tips"], case["sites"]
        lanes = case.get("lanes") or next(b for b in (4, 8, 16, 32) if case["states"] <= b)
        b = (2 * n - 1) * sites * lanes / 8.0 + 8.0 * sites
        # a lane operation per site and node; a pass over the states for a median
        return {"bytes": b, "flops": 0.0 if kind == "fitch" or lanes == 4 else 2.0 * case["states"] * n * sites}
    if kind == "mlp":
        net = 2.0 * (64 * 256 + 2 * 256 * 256 + 256)
        return {"bytes": 4.0 * 65 * case["rows"] + 8.0 * 148481,
                "flops": net * (case["rows"] + 3.0 * case["batch"] * case["steps"])}
    if kind == "batch":
        n, v = case["tips"], case["variants"]
        p = (case["min_patterns"] + case["max_patterns"]) / 2.0 * v
        return {"bytes": p * (n + 16.0), "flops": p * n * 0.5 * 2.0 * (4 * 20 * 20 + 61 * 61)}
    n, p, r = case["tips"], float(case["patterns"]), case["rates"]
    node = r * (2 * 2 * 16 + 4.0)
    if kind in ("prune", "prune_host"):
        return {"bytes": p * (n + 16.0), "flops": (n - 1) * p * node}
    if kind == "fit":
        return {"bytes": p * (n + 8.0), "flops": case["models"] * (n - 1) * p * node}
    if kind == "fold":   # each internal vector written once and read once
        vec = r * 4.0 * case["precision"] / 8 + 4
        return {"bytes": p * (n + 16.0 + 2 * (n - 1) * vec), "flops": (n - 1) * p * node}
    moves = 4.0 * (n - 2) * (n - 3)
    pool = 2.0 * (2 * n - 3) * p * r * 68      # both directions of every edge
    move = p * r * 80.0                        # a rebuilt vector, moved half a branch, and a dot product
    if kind == "scan":
        return {"bytes": p * (n + 8.0) + 8 * moves, "flops": pool + moves * move}
    return {"bytes": p * (n + 8.0) + 256 * moves, "flops": 4 * pool + case["moves"] * n * move}


# ---- the same numbers in 64 bits ---------------------------------------------------

def _q_gtr(co, pi):
    q = np.zeros((4, 4))
    iu = np.triu_indices(4, 1)
    q[iu] = np.append(co, 1.0)
    q = (q + q.T) * pi
    np.fill_diagonal(q, -q.sum(1))
    return q / -(np.diag(q) * pi).sum()


def _site_lnl(tr, q, pi, rates, probs, table, codes):
    """Pattern log-likelihoods by plain FP64 pruning (torch, on the GPU)."""
    n, s, r = tr.n_tips, len(pi), len(rates)
    t = torch.as_tensor(tr.brlen)[:, None] * torch.as_tensor(rates)
    P = torch.linalg.matrix_exp(t[:, :, None, None] * torch.as_tensor(q)).to(DEV)    # [branch, R, S, S]
    tab = torch.as_tensor(table, device=DEV)
    root = (torch.as_tensor(pi, device=DEV) * torch.as_tensor(probs, device=DEV)[:, None])
    out = []
    step = max(4096, (1 << 22) // (s * r))
    for p0 in range(0, codes.shape[1], step):
        part = codes[:, p0:p0 + step].long()
        m = part.shape[1]
        scale = torch.zeros(m, dtype=torch.float64, device=DEV)
        live = {}
        for k in range(n - 1):
            x = None
            for c in (int(tr.left[k]), int(tr.right[k])):
                if c < n:
                    rows = torch.matmul(tab, P[c].transpose(1, 2))                   # [R, codes, S]
                    y = rows[:, part[c]]
                else:
                    y = torch.matmul(live.pop(c), P[c].transpose(1, 2))
                x = y if x is None else x * y
            top = x.amax(dim=(0, 2))
            scale += torch.log(top)
            live[n + k] = x / top[None, :, None]
        out.append(torch.log((live.pop(2 * n - 2) * root[:, None, :]).sum(dim=(0, 2))) + scale)
    return torch.cat(out)


def exact(case, seed):
    kind = case["kind"]
    if kind in ("prune", "prune_host", "fit", "fold"):
        rng, gen, tr, par, codes, w = _dna_problem(case, seed)
        table = _dna_table()
        if kind == "fit":
            return torch.stack([(_site_lnl(tr, _q_gtr(*m[:2]), *m[1:], table, codes) * w).sum()
                                for m in _fit_models(rng, par, case["models"])])
        site = _site_lnl(tr, _q_gtr(*par[:2]), *par[1:], table, codes)
        lnl = (site * w).sum()
        if kind == "prune":
            return lnl.reshape(1), site
        return (float(lnl), site) if kind == "prune_host" else (-float(lnl), site)
    if kind == "batch":
        sites, total = [], []
        for tr, q, pi, r, p, codes, w, n in _variants(case, seed):
            sites.append(_site_lnl(tr, q, pi, r, p, _state_table(len(pi)), codes))
            total.append((sites[-1] * w).sum())
        return torch.stack(total), torch.cat(sites)
    if kind == "mlp":
        params, x, _ = _network(case, seed)
        x = x.double()
        sd = x.std(dim=0, unbiased=False)
        h = (x - x.mean(dim=0)) / sd
        at = 0
        for rows, cols in ((256, 64), (256, 256), (256, 256), (1, 256)):
            wgt = torch.as_tensor(params[at:at + rows * cols], device=DEV).double().reshape(rows, cols)
            h = h @ wgt.T
            at += rows * cols + rows
            if rows > 1:
                h = torch.nn.functional.gelu(h)
        return h[:, 0], None
    return None   # whole numbers; or every neighbour of a tree rescored, which takes minutes
