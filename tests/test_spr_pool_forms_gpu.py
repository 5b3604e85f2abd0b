"""GPU: the SPR pool made with and without its mid-edge vectors, the float-pair
eigen products and state profiles, and the Fitch sets kept as bit planes, at
rate-class counts with idle lanes, odd pattern counts and fractional weights."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import spr_oracle as SO
from phylocaml_gb300 import mlmodel as M, spr, synth, tree as T

pytestmark = pytest.mark.gpu


def problem(ctx, n, n_pat, k, seed, fraction, gaps=0.0):
    import torch
    rng = np.random.default_rng(seed)
    tr = T.yule(n, rng, 0.2)
    spec = synth.random_gtr_spec(rng, 0.7, k)
    q, pi, rates, probs = synth.host_model(spec)
    states = synth.simulate_sites(tr, q, pi, rates, probs, n_pat, rng)
    pats = (np.uint8(1) << states).astype(np.uint8)
    pats[rng.random(pats.shape) < gaps] = 15
    w = rng.integers(1, 300, size=n_pat) * fraction
    dev = torch.device("cuda:0")
    return dict(tr=tr, q=q, pi=pi, rates=rates, probs=probs, model=M.create(spec, ctx), pats=pats, w=w,
                tips=torch.from_numpy(pats).to(dev), wd=torch.from_numpy(w).to(dev),
                table=synth.dna_code_table())


def engine(d, ctx, prec):
    e = spr.SprEngine(d["tips"], d["pats"].shape[1], d["model"], d["table"], d["wd"], prec, ctx)
    e.set_tree(d["tr"])
    return e


@pytest.mark.parametrize("prec,k,n_pat,fraction", [(48, 1, 37, 0.3), (48, 3, 257, 0.3), (48, 8, 64, 1.0),
                                                   (32, 5, 33, 0.3), (64, 4, 31, 0.3)])
def test_vectors_added_later_score_the_same(ctx, prec, k, n_pat, fraction):
    """A few moves (their own mid-edge vectors only), then every move (the rest
    added), then TBR, against a pool made with all of them at once.  The same
    site values in other groups: the sums agree to the pairs' 1e-12."""
    d = problem(ctx, 9, n_pat, k, 5 + k, fraction)
    few = np.array([3, 100, 3, 167])
    e = engine(d, ctx, prec)
    want = e.scan().cpu().numpy()
    tbr = e.tbr_scan().cpu().numpy()
    e.set_tree(d["tr"])
    assert np.allclose(e.score(few), want[few], rtol=1e-12, atol=0)
    assert np.allclose(e.scan().cpu().numpy(), want, rtol=1e-12, atol=0)
    e.set_tree(d["tr"])
    assert np.allclose(e.score(np.arange(len(want))), want, rtol=1e-12, atol=0)
    e.set_tree(d["tr"])
    e.lnl()
    assert np.array_equal(e.tbr_scan().cpu().numpy(), tbr)
    cur = e.get_tree()
    adj = SO.unroot(cur.left, cur.right, cur.brlen)
    mv = e.moves()
    tol = {64: 1e-10, 48: 1e-9}.get(prec)
    for i in few:
        exp = SO.lnl(SO.apply_move(adj, *mv[i]), 9, d["q"], d["pi"], d["rates"], d["probs"], d["pats"],
                     d["table"], d["w"])
        assert abs(want[i] - exp) <= (tol * abs(exp) if tol else 2e-6 * d["w"].sum())
    e.close()


@pytest.mark.parametrize("k,n_pat,fraction,gaps", [(1, 401, 0.3, 0.0), (3, 400, 1.0, 0.5), (4, 1000, 0.3, 0.1)])
def test_pair_profiles_and_lengths_follow_fp64(ctx, k, n_pat, fraction, gaps):
    """Features: profiles are means of ratios of values rounded to float (2^-24
    each) stored as float: within 1e-6 of the FP64 engine's.  Lengths: the eigen
    products round to the same floats up to the vectors' own last bits, so a
    Newton round ends at the same likelihood to 1e-9."""
    d = problem(ctx, 12, n_pat, k, 40 + k, fraction, gaps)
    got, lnl = [], []
    for prec in (48, 64):
        e = engine(d, ctx, prec)
        got.append(e.features().cpu().numpy())
        lnl.append(e.optimize(1, 1e-4))
        e.close()
    assert np.abs(got[0] - got[1]).max() <= 1e-6
    assert abs(lnl[0] - lnl[1]) <= 1e-9 * abs(lnl[1])


@pytest.mark.parametrize("n,n_pat,fraction", [(5, 1, 1.0), (6, 33, 2.0), (7, 4133, 1.0), (1400, 40, 9.0)])
def test_fitch_planes(ctx, n, n_pat, fraction):
    """Parsimony lengths are whole numbers and exact: a lone pattern, a second
    word, more words than a CTA, weights beyond the planes held in registers,
    and a tree whose lengths do not fit in shared memory."""
    d = problem(ctx, n, n_pat, 1, n, fraction, 0.05)
    e = engine(d, ctx, 48)
    if n > 100:
        e.set_join_distance(1)
    lens, total = e.fitch()
    cur = e.get_tree()
    adj = SO.unroot(cur.left, cur.right, cur.brlen)
    masks = spr.code_masks(d["table"])
    assert total == SO.fitch_length(adj, n, d["pats"], masks, d["w"])
    mv, lens = e.moves(), lens.cpu().numpy()
    for i in range(0, len(mv), max(1, len(mv) // 6)):
        assert lens[i] == SO.fitch_length(SO.apply_move(adj, *mv[i]), n, d["pats"], masks, d["w"])
    e.close()


@pytest.mark.parametrize("prec,k,n_pat", [(48, 1, 129), (48, 2, 63), (48, 4, 33), (48, 8, 17), (32, 3, 40), (64, 2, 65)])
def test_more_moves_than_a_window(ctx, prec, k, n_pat):
    """Prunes of up to 74 moves, summed over the warps 64 at a time, against the
    same moves scored a few to a prune and against the oracle."""
    d = problem(ctx, 40, n_pat, k, 70 + k, 1.0)
    e = engine(d, ctx, prec)
    got = e.scan().cpu().numpy()
    rng = np.random.default_rng(k)
    some = rng.choice(len(got), 40, replace=False)
    assert np.allclose(e.score(some), got[some], rtol=1e-12, atol=0)
    cur = e.get_tree()
    adj = SO.unroot(cur.left, cur.right, cur.brlen)
    mv = e.moves()
    tol = {64: 1e-10, 48: 1e-9}.get(prec)
    for i in some[:8]:
        exp = SO.lnl(SO.apply_move(adj, *mv[i]), 40, d["q"], d["pi"], d["rates"], d["probs"], d["pats"],
                     d["table"], d["w"])
        assert abs(got[i] - exp) <= (tol * abs(exp) if tol else 2e-6 * d["w"].sum())
    e.close()


def test_groups_of_pattern_blocks(ctx):
    """Enough moves and patterns that a CTA walks several blocks: the partial
    sums are added up in place, and agree with the moves scored by themselves."""
    d = problem(ctx, 120, 80000, 1, 3, 1.0)
    e = engine(d, ctx, 32)
    got = e.scan().cpu().numpy()
    assert len(got) * -(-80000 // 128) * 8 > 256 << 20
    some = np.random.default_rng(0).choice(len(got), 30, replace=False)
    assert np.allclose(e.score(some), got[some], rtol=1e-12, atol=0)
    e.close()
