"""GPU: four-state medians over leaves kept as codes.  Every mix of leaf and
internal neighbours, 1 to 8 rate classes, code tables on both sides of the
shared-memory limit, ragged pattern counts and reused handles, against the
FP64 recursion in numpy; node costs and their reuse; bad codes found by every
call that synchronises."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import mlmodel_oracle as O
from phylocaml_gb300 import _native, likelihood_c as L, mlmodel as M, synth

pytestmark = pytest.mark.gpu

# eps of the storage type times a few roundings per entry and neighbour
REL = {32: 2e-6, 64: 1e-12}


def _site(x, pi, probs):
    return np.log(np.einsum("r,i,nri->n", probs, pi, x))


@pytest.mark.parametrize("prec", [32, 64])
@pytest.mark.parametrize("rates,n_codes,n_pat", [(1, 16, 1), (2, 16, 255), (3, 16, 513), (4, 16, 1000),
                                                 (5, 40, 777), (8, 256, 301), (4, 256, 129)])
def test_medians_of_leaves_and_nodes(ctx, prec, rates, n_codes, n_pat):
    rng = np.random.default_rng(rates * 1000 + n_pat)
    spec = synth.random_gtr_spec(rng, 0.5, rates)
    model = M.create(spec, ctx)
    q, pi, r, probs = synth.host_model(spec)
    table = (rng.random((n_codes, 4)) < 0.5).astype(np.float64)
    table[:, 0] = 1.0
    w = rng.integers(1, 9, n_pat).astype(np.float64)
    codes = rng.integers(0, n_codes, (4, n_pat)).astype(np.uint8)
    t = [0.11, 0.0, 0.7, 0.05, 0.2]
    P = O.pmatrices(q, pi, r, t)                                   # [5][R][4][4]
    up = lambda k, x: np.einsum("rij,nrj->nri", P[k], x)           # noqa: E731
    leafx = [np.repeat(table[c][:, None, :], rates, axis=1) for c in codes]
    lk = L.LkModel(model, table, n_pat, w, prec, ctx)
    try:
        leaf = [lk.leaf(c, t[k]) for k, c in enumerate(codes)]
        ab = L.median_2(lk, None, leaf[0], leaf[1])                # leaf, leaf
        ab.set_brlen(t[4])
        xab = up(0, leafx[0]) * up(1, leafx[1])
        cases = [([ab, leaf[2]], up(4, xab) * up(2, leafx[2])),    # node, leaf
                 ([leaf[2], ab], up(4, xab) * up(2, leafx[2])),
                 ([ab], up(4, xab)),
                 ([leaf[3]], up(3, leafx[3])),
                 ([leaf[2], ab, leaf[3]], up(2, leafx[2]) * up(4, xab) * up(3, leafx[3]))]
        reuse = None
        for nbrs, x in cases * 2:                                  # the same handle over and over
            reuse = lk.median(reuse, *nbrs)
            internal = [ab] if any(n is ab for n in nbrs) else []
            # a pattern's lnL is at its root; costs carry what was normalised away
            cost, site = reuse.root_cost(site_lnl=True)
            exp = _site(x, pi, probs)
            total = cost + L.cost(reuse) + sum(L.cost(n) for n in internal)
            scale = np.maximum(np.abs(exp), 1.0)
            assert np.all(np.abs(site - exp) <= REL[prec] * 4 * scale)
            assert abs(total + float((w * exp).sum())) <= REL[prec] * 4 * float((w * scale).sum())
        assert L.cost(leaf[0]) == 0.0
        assert np.all(lk.costs([leaf[1], leaf[2]]) == 0.0)
        # a leaf's own likelihood, and the leaf as a neighbour afterwards
        got = leaf[3].root_cost(site_lnl=True)[1]
        assert np.all(np.abs(got - _site(leafx[3], pi, probs)) <= 1e-6)
        again = L.median_1(lk, None, leaf[3])
        assert np.all(np.abs(again.root_cost(site_lnl=True)[1] - _site(up(3, leafx[3]), pi, probs))
                      <= REL[prec] * 40)
    finally:
        lk.close()


def test_fractional_weights_and_bad_codes(ctx):
    rng = np.random.default_rng(3)
    spec = synth.random_gtr_spec(rng, 0.5)
    model = M.create(spec, ctx)
    w = rng.random(400) * 3
    table = synth.dna_code_table()
    good = rng.integers(1, 16, 400).astype(np.uint8)
    lk = L.LkModel(model, table, 400, w, 64, ctx)
    one = L.LkModel(model, table, 400, np.ones(400), 64, ctx)
    try:
        for m, wt in ((lk, w), (one, np.ones(400))):
            a, b = m.leaf(good, 0.3), m.leaf(good[::-1].copy(), 0.1)
            n = L.median_2(m, None, a, b)
            cost, site = n.root_cost(site_lnl=True)
            assert abs(cost + L.cost(n) + float((wt * site).sum())) <= 1e-11 * abs(float((wt * site).sum()))
        bad = good.copy()
        bad[399] = 16
        for call in (lambda t: L.cost(t), lambda t: lk.costs([t]), lambda t: t.root_cost(),
                     lambda t: L.cost(L.median_1(lk, None, t))):
            t = lk.leaf(bad, 0.1)
            with pytest.raises(_native.NativeError):
                call(t)
        t = lk.leaf(bad, 0.1)
        t = lk.leaf(good, 0.2, o=t)                    # overwritten before anything read it
        assert L.cost(t) == 0.0
        lk.leaf(bad, 0.1).close()
        assert L.cost(lk.leaf(good, 0.1)) == 0.0
    finally:
        lk.close()
        one.close()
