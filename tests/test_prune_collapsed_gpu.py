"""GPU: pruning with small subtrees collapsed into leaves (two tips from 512
patterns on, three from 8,192, at 16 codes) against the walk over every node,
which the same patterns take in slices below those counts, and against the
FP64 oracle; trees of few tips, branches that force rescaling inside a
collapsed subtree, and codes outside the table."""
from __future__ import annotations

import numpy as np
import pytest

import oracle as orc
from oracle import mlmodel_oracle as O
from phylocaml_gb300 import _native, likelihood as Lk, mlmodel as M, synth, tree as T

pytestmark = pytest.mark.gpu

# sums of a few hundred terms rounded at 2^-48 (pairs) and 2^-53 (FP64); the
# FP32 form does the same operations on the same values
REL = {32: 0.0, 48: 1e-12, 64: 1e-13}


def _case(n_tips, n_pat, seed, brlen=0.1, rates=4):
    rng = np.random.default_rng(seed)
    tr = T.yule(n_tips, rng, brlen) if n_tips > 4 else T.caterpillar(n_tips, brlen)
    spec = synth.random_gtr_spec(rng, 0.5, rates)
    states = synth.jc_states(tr, n_pat, rng)
    masks = (np.uint8(1) << states).astype(np.uint8)
    synth.inject_ambiguity(masks, 0.05, rng)
    return tr, spec, masks, rng.integers(1, 5, n_pat).astype(np.float64)


def _site(tr, model, codes, w, prec, ctx):
    return Lk.tree_lnl(tr, model, codes, synth.dna_code_table(), w, prec, ctx, site_lnl=True)


@pytest.mark.parametrize("prec", [32, 48, 64])
@pytest.mark.parametrize("n_tips,rates", [(2, 4), (3, 4), (4, 1), (7, 4), (40, 3), (61, 5)])
def test_collapsed_equals_every_node(ctx, prec, n_tips, rates):
    n_pat = 8209
    tr, spec, codes, w = _case(n_tips, n_pat, 10 * n_tips + rates, rates=rates)
    model = M.create(spec, ctx)
    lnl, site = _site(tr, model, codes, w, prec, ctx)            # three tips to a leaf
    for step in (8191, 511):                                     # two, none
        for p0 in range(0, n_pat, step):
            part = np.ascontiguousarray(codes[:, p0:p0 + step])
            got = _site(tr, model, part, w[p0:p0 + step], prec, ctx)[1]
            ref = site[p0:p0 + step]
            assert np.all(np.abs(got - ref) <= REL[prec] * np.abs(ref))
    assert abs(lnl - float(np.sum(site * w))) <= 1e-12 * abs(lnl)


@pytest.mark.parametrize("brlen", [1e-9, 1e-7, 3.0])
def test_rescaling_inside_a_collapsed_subtree(ctx, brlen):
    # differing tips on branches this short make a cherry's vector fall below
    # the rescaling threshold
    tr, spec, codes, w = _case(30, 9000, 5, 0.2)
    tr = T.RootedTree(tr.left, tr.right, np.full_like(tr.brlen, brlen))
    q, pi, rates, probs = synth.host_model(spec)
    P = O.pmatrices(q, pi, rates, tr.brlen)
    if brlen < 1:
            # U exp(Dt) Ui leaves short branches' off-diagonal entries an
            # absolute error of 1e-16, 1.2e-9 of this lnL at 1e-9: the series
            # to third order has them to 1e-16 of themselves (and an
            # effective length below 1e-10 is the identity)
            t = np.where(rates * brlen < 1e-10, 0.0, rates * brlen)
            X = q[None] * t[:, None, None]
            P[:] = np.eye(4) + X + X @ X / 2 + X @ X @ X / 6
    exp = orc.prune_lnl(tr.left, tr.right, P, pi, probs, codes, synth.dna_code_table(), w)
    model = M.create(spec, ctx)
    for prec, rel in ((48, 1e-9), (64, 1e-9)):
        got = Lk.tree_lnl(tr, model, codes, synth.dna_code_table(), w, prec, ctx)
        assert abs(got - exp) <= rel * abs(exp)


def test_many_models_and_bad_codes(ctx):
    tr, spec, codes, w = _case(50, 8300, 6)
    rng = np.random.default_rng(9)
    models = [M.create(synth.random_gtr_spec(rng, 0.3 + 0.1 * k, 4), ctx) for k in range(5)]
    got = Lk.tree_lnl_models(tr, models, codes, synth.dna_code_table(), w, 48, ctx)
    for m, v in zip(models, got):
        assert v == Lk.tree_lnl(tr, m, codes, synth.dna_code_table(), w, 48, ctx)
    codes[7, 8299] = 16
    with pytest.raises(_native.NativeError) as e:
        Lk.tree_lnl(tr, models[0], codes, synth.dna_code_table(), w, 48, ctx)
    assert e.value.status == 1
