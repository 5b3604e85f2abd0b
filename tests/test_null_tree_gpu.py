"""GPU: a tree without child arrays is an argument error of the cost-matrix and
Fitch calls, also right after a tree of the same size."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from phylocaml_gb300 import _native, costmatrix, tree as T

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("call", ["pgpu_fitch_tree_dev", "pgpu_tcm_tree_dev", "pgpu_tcm_tree_wide_dev"])
def test_tree_without_children(ctx, call):
    import torch
    tr, n, words = T.caterpillar(6, 0.1), 6, 4
    tips = torch.full((n, words), 0x11111111 if call == "pgpu_tcm_tree_dev" else 0x01010101, dtype=torch.int32, device="cuda:0")
    sets, total = torch.zeros((n - 1, words), dtype=torch.int32, device="cuda:0"), torch.zeros(1, dtype=torch.int64,
                                                                                              device="cuda:0")
    tcm = np.ones((5, 5), np.int32) - np.eye(5, dtype=np.int32)
    m4 = costmatrix.CostMatrix(np.ascontiguousarray(tcm[:4, :4]), "general")
    mode = {"pgpu_fitch_tree_dev": lambda: (8,),
            "pgpu_tcm_tree_dev": lambda: (m4.table.ctypes.data,),
            "pgpu_tcm_tree_wide_dev": lambda: (8, tcm.ctypes.data, 5, costmatrix.MODES["general"], 1)}[call]()
    sites = 8 if call != "pgpu_tcm_tree_dev" else 16
    torch.cuda.synchronize()
    t, keep = _native.make_tree(tr.left, tr.right)

    def run(tree):
        ctx.call(call, C.byref(tree), tips.data_ptr(), words, None, sites, *mode, sets.data_ptr(), None,
                 total.data_ptr())

    run(t)
    ctx.synchronize()
    for missing in ("left", "right"):
        bad = _native.PgpuTree(t.n_tips, t.left, t.right, None)
        setattr(bad, missing, None)
        with pytest.raises(_native.NativeError) as e:
            run(bad)
        assert e.value.status == 1
    run(t)
    ctx.synchronize()
    del keep
