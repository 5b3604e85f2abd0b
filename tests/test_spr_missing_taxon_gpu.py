"""GPU: the branch above a taxon without any data does not change the
likelihood, and what a Newton round makes of its length is decided by the
rounding of sums that cancel.  The pair form takes those from FP64, so its
lengths stay those of the FP64 form; they agree to the 3e-7 that a last bit of
the float sums is worth, a few times over."""
from __future__ import annotations

import numpy as np
import pytest

from phylocaml_gb300 import mlmodel as M, spr, synth, tree as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed", range(8))
def test_lengths_follow_fp64(ctx, seed):
    import torch
    rng = np.random.default_rng(seed)
    n, n_pat = 9, 300
    tr = T.yule(n, rng, 0.1)
    model = M.create(synth.random_gtr_spec(rng, 0.5, 4), ctx)
    codes = (np.uint8(1) << synth.jc_states(tr, n_pat, rng)).astype(np.uint8)
    codes[rng.integers(0, n)] = 15
    dev = torch.device("cuda:0")
    cd, w = torch.from_numpy(codes).to(dev), torch.from_numpy(rng.integers(1, 4, n_pat).astype(np.float64)).to(dev)
    got = {}
    for prec in (48, 64):
        e = spr.SprEngine(cd, n_pat, model, synth.dna_code_table(), w, prec, ctx)
        e.set_tree(tr)
        e.optimize(1, 1e-4)
        got[prec] = e.lengths()[0]
        e.close()
    np.testing.assert_allclose(got[48], got[64], rtol=1e-6)
