"""GPU: the wide cost-matrix kernel's packed rows at the sizes where they
change shape -- state counts around each row width, costs around the
16-bit form's limit, site counts around a warp -- bit-exact against the
restatement of the median rules."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import tcm_oracle as TO
from phylocaml_gb300 import costmatrix as CM, tree as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("S,n_sites,top", [
    (2, 1, 16383), (7, 31, 16384), (8, 33, 16383), (9, 64, 16384), (16, 35, 16383), (16, 3, 1 << 25),
    (17, 32, 16383), (24, 65, 16384), (25, 29, 16383), (25, 97, 1 << 24), (32, 40, 1 << 25), (32, 30, 16383)])
@pytest.mark.parametrize("mode", ["general", "metric"])
def test_rows_against_restatement(ctx, S, n_sites, top, mode):
    rng = np.random.default_rng(100 * S + n_sites)
    n = 2 if n_sites == 3 else 21
    tr = T.yule(n, rng, 0.1)
    tcm = rng.integers(0, top + 1, (S, S)).astype(np.int32)
    tcm[rng.integers(S), rng.integers(S)] = top           # the limit itself occurs
    tcm[:, rng.integers(S)] //= 1000                      # and so do ties at small costs
    codes = np.int64(1) << rng.integers(0, S, (n, n_sites))
    codes |= np.where(rng.random(codes.shape) < 0.4, np.int64(1) << rng.integers(0, S, codes.shape), 0)
    codes[rng.random(codes.shape) < 0.1] = (1 << S) - 1   # every state
    cm = CM.CostMatrix(tcm, mode=mode, symmetric=False)
    w = rng.integers(1, 9, n_sites).astype(np.uint32)
    lb = next(b for b in (8, 16, 32) if S <= b)
    node, site, total = TO.tree_cost_direct(tr.left, tr.right, codes, cm.tcm, CM.MODES[mode], False, w)
    r = cm.tree_cost(tr, codes.astype(np.uint32), w, ctx, lane_bits=lb)
    assert np.array_equal(r.states().astype(np.int64), node)
    assert np.array_equal(r.site_cost.astype(np.int64), site) and r.total == total
