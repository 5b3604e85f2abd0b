"""GPU: pruning from host arrays at the sizes where the call changes its way:
data and results that just fit and just do not fit the staging blocks, and the
number of models from which the eigen systems are solved on the GPU."""
from __future__ import annotations

import numpy as np
import pytest

from phylocaml_gb300 import likelihood as Lk, mlmodel as M, synth, tree as T

pytestmark = pytest.mark.gpu


def case(n_tips, n_pat, seed):
    rng = np.random.default_rng(seed)
    tr = T.yule(n_tips, rng, 0.1)
    states = synth.jc_states(tr, n_pat, rng)
    return tr, (np.uint8(1) << states).astype(np.uint8), rng.integers(1, 5, n_pat).astype(np.float64), rng


@pytest.mark.parametrize("prec", [32, 48, 64])
@pytest.mark.parametrize("n_tips,most", [
    (32, 3265),     # codes and weights on either side of 128 KB
    (8, 16385),     # site results on either side of 128 KB
])
def test_sizes_around_the_staging_blocks(ctx, prec, n_tips, most):
    """The same patterns in calls of one pattern less give the same bits."""
    tr, codes, w, rng = case(n_tips, most, 11 + n_tips)
    model = M.create(synth.random_gtr_spec(rng, 0.5, 4), ctx)
    table = synth.dna_code_table()
    lnl, site = Lk.tree_lnl(tr, model, codes, table, w, prec, ctx, site_lnl=True)
    assert abs(lnl - float(np.sum(site * w))) <= 1e-12 * abs(lnl)
    for n in (most - 1, most - 2, most - 17):
        part = np.ascontiguousarray(codes[:, :n])
        for weights in (w[:n], None):
            got, s = Lk.tree_lnl(tr, model, part, table, weights, prec, ctx, site_lnl=True)
            assert np.array_equal(s, site[:n])
            want = float(np.sum(site[:n] * (w[:n] if weights is not None else 1.0)))
            assert abs(got - want) <= 1e-12 * abs(want)


@pytest.mark.parametrize("count", [1, 24, 25, 40])
def test_models_around_the_eigen_rule(ctx, count):
    """Eigen systems from the host (up to 24 models) and from the GPU: both are
    Jacobi rotations in FP64, so log-likelihoods agree to 1e-11."""
    tr, codes, w, rng = case(20, 700, 3)
    models = [M.create(synth.random_gtr_spec(rng, 0.3 + 0.02 * k, 4), ctx) for k in range(count)]
    got = Lk.tree_lnl_models(tr, models, codes, synth.dna_code_table(), w, 64, ctx)
    for m, v in zip(models, got):
        one = Lk.tree_lnl(tr, m, codes, synth.dna_code_table(), w, 64, ctx)
        assert abs(v - one) <= 1e-11 * abs(one)
