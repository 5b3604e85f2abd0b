"""GPU: batched scoring of an alphabet far smaller than its padding, on trees
that leave stack slots unused, every code holding a state, so that every score
is a number; against the FP64 form, with one and two rate classes per pass.

TF32 keeps 11 bits: an internal child's product P x, a sum of non-negative
terms, is off by at most 2^-11 for each of the two operands (a bit over, for
their product), so a pattern's log-likelihood by 2.001 x 2^-11 for each of the
tree's internal children."""
from __future__ import annotations

import numpy as np
import pytest

from phylocaml_gb300 import mlmodel as M, synth, tree as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,R,n_codes,tips", [(3, 2, 8, 128), (2, 4, 3, 64), (9, 2, 200, 16)])
@pytest.mark.parametrize("shape", ["balanced", "yule"])
def test_small_alphabets(ctx, S, R, n_codes, tips, shape):
    import torch
    from phylocaml_gb300.batch import Batch, Options, Variant, device_codes
    rng = np.random.default_rng(S * 100 + R)
    dev = torch.device("cuda:0")
    vs, most = [], []
    for k, n_pat in enumerate((300, 128, 1)):
        tr = T.balanced(tips, 0.1) if shape == "balanced" else T.yule(tips + k, rng, 0.1)
        ex = np.triu(rng.lognormal(0.0, 1.0, (S, S)), 1)
        pi = rng.dirichlet(np.full(S, 5.0))
        table = (rng.random((n_codes, S)) < 0.3).astype(np.float64)
        table[np.arange(n_codes), np.arange(n_codes) % S] = 1.0
        inner = int(np.sum(tr.left >= tr.n_tips) + np.sum(tr.right >= tr.n_tips))
        wh = rng.integers(1, 4, n_pat).astype(np.float64)
        most.append(inner * 2.001 * 2.0 ** -11 * wh.sum())
        vs.append(Variant(tr, synth.normalize_q((ex + ex.T) * pi[None, :], pi), pi, M.gamma_rates(0.7, R),
                          np.full(R, 1.0 / R), table,
                          device_codes(rng.integers(0, n_codes, (tr.n_tips, n_pat)).astype(np.uint8), dev),
                          torch.from_numpy(wh).to(dev), n_pat))
    got = []
    for pairs in (True, False):
        b = Batch(vs, ctx, Options(pairs, "cost"))
        try:
            got.append(b.run())
            f64 = b.run_fp64(sample=300)
        finally:
            b.close()
    assert np.all(np.isfinite(f64)) and np.all(np.isfinite(got))
    assert np.all(np.abs(got[0] - f64) <= most), (got[0] - f64, most)
    np.testing.assert_allclose(got[0], got[1], rtol=1e-12)
