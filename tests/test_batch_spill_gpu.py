"""GPU: batched scoring where a tile's vectors do not fit its half of tensor
memory and go through global memory, and where the ring of staged blocks has
two, three or four slots or leaves room for one CTA per SM, against the FP64
form.  The same trees with one and two rate classes per pass keep their vectors
in different places and give the same scores."""
from __future__ import annotations

import numpy as np
import pytest

from phylocaml_gb300 import mlmodel as M, synth, tree as T

pytestmark = pytest.mark.gpu

# TF32 operands are rounded to 11 bits without bias: 5e-7 of the score on the
# workload's shapes; a vector in the wrong place is off by whole nats a pattern
REL = 1e-4


def variant(rng, tr, S, R, n_codes, n_pat):
    import torch
    from phylocaml_gb300.batch import Variant, device_codes
    ex = np.triu(rng.lognormal(0.0, 1.0, (S, S)), 1)
    pi = rng.dirichlet(np.full(S, 5.0))
    q = synth.normalize_q((ex + ex.T) * pi[None, :], pi)
    rates = M.gamma_rates(0.7, R) if R > 1 else np.ones(1)
    table = np.vstack([np.eye(S), (rng.random((n_codes, S)) < 0.3) | np.eye(n_codes, S, dtype=bool)])[:n_codes]
    codes = rng.integers(0, n_codes, (tr.n_tips, n_pat)).astype(np.uint8)
    w = rng.integers(1, 4, n_pat).astype(np.float64)
    dev = torch.device("cuda:0")
    return Variant(tr, q, pi, rates, np.full(R, 1.0 / R), table.astype(np.float64), device_codes(codes, dev),
                   torch.from_numpy(w).to(dev), n_pat)


@pytest.mark.parametrize("S,R,n_codes,tips", [
    (61, 1, 62, 64),     # 3 slots, nested spills, ring of 3
    (50, 2, 51, 32),     # D wider than a slot, one class per pass
    (56, 1, 120, 16),    # blocks that leave room for one CTA per SM
    (20, 4, 21, 128),    # two classes per pass, 4 slots, ring of 4
    (30, 2, 31, 64),     # two classes per pass, 3 slots
    (24, 4, 140, 32),    # blocks too large for two classes per pass
    (61, 1, 100, 16),    # ring of 2
    (3, 2, 8, 128),      # more slots than any tree takes
])
@pytest.mark.parametrize("shape", ["balanced", "yule"])
def test_spilled_vectors(ctx, S, R, n_codes, tips, shape):
    from phylocaml_gb300.batch import Batch, Options
    rng = np.random.default_rng(S * 10 + R)
    vs = [variant(rng, T.balanced(tips, 0.1) if shape == "balanced" else T.yule(tips + k, rng, 0.1), S, R, n_codes, p)
          for k, p in enumerate((300, 128, 1))]
    got = []
    for pairs in (True, False):
        b = Batch(vs, ctx, Options(pairs, "cost"))
        try:
            got.append(b.run())
            f64 = b.run_fp64(sample=300)
        finally:
            b.close()
    np.testing.assert_allclose(got[0], f64, rtol=REL)   # a code without states makes both forms NaN
    np.testing.assert_allclose(got[0], got[1], rtol=1e-12)
