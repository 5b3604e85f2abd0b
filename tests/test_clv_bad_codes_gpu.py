"""GPU: a four-state leaf with a code outside the table is reported by the next
call that checks the context's errors, whether or not anything has read the
leaf, on both sides of the size that goes through the staging blocks; reported
once, and such a code then counts as code 0."""
from __future__ import annotations

import numpy as np
import pytest

from phylocaml_gb300 import _native, fitch, likelihood_c as L, mlmodel as M, synth, tree as T

pytestmark = pytest.mark.gpu


def fails(call):
    with pytest.raises(_native.NativeError) as e:
        call()
    assert e.value.status == 1   # PGPU_ERR_ARG, as for any code outside a table


@pytest.mark.parametrize("n_pat", [7, 40_000, (1 << 20) + 5])
@pytest.mark.parametrize("at", [0, -1])
def test_reported_without_a_reader(native_lib, n_pat, at):
    rng = np.random.default_rng(n_pat)
    good = rng.integers(1, 16, n_pat).astype(np.uint8)
    bad = good.copy()
    bad[at] = 16
    with _native.Context(0) as ctx:
        lk = L.LkModel(M.create(synth.random_gtr_spec(rng, 0.5), ctx), synth.dna_code_table(), n_pat, None, 64, ctx)
        leaf = lk.leaf(bad, 0.1)
        fails(ctx.synchronize)
        ctx.synchronize()                       # once
        other = lk.leaf(bad, 0.1)
        words = np.full((4, 1), 0x11111111, np.uint32)
        fails(lambda: fitch.fitch_tree(T.caterpillar(4, 0.1), words, 8, ctx=ctx))   # another call of the context
        # the code then counts as code 0 and is no error to read
        zero = good.copy()
        zero[at] = 0
        node = L.median_2(lk, None, leaf, other)
        want = L.median_2(lk, None, lk.leaf(zero, 0.1), lk.leaf(zero, 0.1))
        assert np.array_equal(node.root_cost(site_lnl=True)[1], want.root_cost(site_lnl=True)[1])
        # read, then gone before any check
        leaf = lk.leaf(bad, 0.3)
        L.median_1(lk, node, leaf)
        leaf.close()
        fails(ctx.synchronize)
        ctx.synchronize()
        lk.close()
