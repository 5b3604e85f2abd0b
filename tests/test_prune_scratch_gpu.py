"""GPU: pruning where the device has no room for its tables of collapsed
subtrees or for the leaf indexes of all patterns: in pieces and with less
collapsed, from device codes, host codes in several chunks and for several
models, the same site log-likelihoods come out."""
from __future__ import annotations

import numpy as np
import pytest

from phylocaml_gb300 import _native, likelihood as Lk, mlmodel as M, synth, tree as T

pytestmark = pytest.mark.gpu

# as where small subtrees are collapsed or not: the FP32 form does the same
# operations, the others round sums of a few hundred terms differently
REL = {32: 0.0, 48: 1e-12, 64: 1e-13}
LIMITS = [1 << 22, 1_600_000, 800_000, 300_000, 100_000, 40_000]
N_TIPS, N_PAT = 12, 120_013   # not a multiple of a tile; two or more chunks of host codes


@pytest.fixture(scope="module")
def case():
    rng = np.random.default_rng(8)
    tr = T.yule(N_TIPS, rng, 0.1)
    masks = (np.uint8(1) << synth.jc_states(tr, N_PAT, rng)).astype(np.uint8)
    synth.inject_ambiguity(masks, 0.05, rng)
    return tr, masks, rng.integers(1, 5, N_PAT).astype(np.float64), synth.dna_code_table()


def limit(ctx, n):
    ctx.call("pgpu_set_scratch_limit", n)


def close(got, want, rel):
    assert np.all(np.abs(got - want) <= rel * np.abs(want))


@pytest.mark.parametrize("prec", [32, 48, 64])
def test_device_codes(native_lib, case, prec):
    import torch
    tr, codes, w, table = case
    ld = (N_PAT + 15) // 16 * 16
    padded = np.zeros((N_TIPS, ld), np.uint8)
    padded[:, :N_PAT] = codes
    dev = torch.device("cuda:0")
    cd, wd = torch.from_numpy(padded).to(dev), torch.from_numpy(w).to(dev)
    lnl, site = torch.zeros(1, dtype=torch.float64, device=dev), torch.zeros(N_PAT, dtype=torch.float64, device=dev)
    with _native.Context(0) as ctx:
        model = M.create(synth.random_gtr_spec(np.random.default_rng(1), 0.5, 4), ctx)

        def run():
            torch.cuda.synchronize()
            before = ctx.launches
            Lk.tree_lnl_dev(tr, model, cd, ld, N_PAT, table, wd, lnl, prec, site, ctx)
            ctx.synchronize()
            return ctx.launches - before, lnl.item(), site.cpu().numpy()

        whole, want, sites = run()
        most = whole
        for n in LIMITS:
            limit(ctx, n)
            k, got, s = run()
            close(s, sites, REL[prec])
            assert abs(got - want) <= max(REL[prec], 1e-15) * abs(want)
            most = max(most, k)
        assert most > whole + 4                      # pieces
        limit(ctx, 4096)                             # not even the P matrices
        with pytest.raises(_native.NativeError) as e:
            run()
        assert e.value.status == 3                   # PGPU_ERR_OOM
        limit(ctx, 0)
        close(run()[2], sites, REL[prec])


@pytest.mark.parametrize("prec", [32, 48])
def test_host_codes_and_models(native_lib, case, prec):
    tr, codes, w, table = case
    with _native.Context(0) as ctx:
        rng = np.random.default_rng(2)
        models = [M.create(synth.random_gtr_spec(rng, 0.3 + 0.2 * k, 4), ctx) for k in range(3)]
        want, sites = Lk.tree_lnl(tr, models[0], codes, table, w, prec, ctx, site_lnl=True)
        each = Lk.tree_lnl_models(tr, models, codes, table, w, prec, ctx)
        for n in (1 << 22, 1_600_000, 1_450_000):     # the codes themselves take 1,440,192 bytes
            limit(ctx, n)
            got, s = Lk.tree_lnl(tr, models[0], codes, table, w, prec, ctx, site_lnl=True)
            close(s, sites, REL[prec])
            assert abs(got - want) <= max(REL[prec], 1e-15) * abs(want)
            close(Lk.tree_lnl_models(tr, models, codes, table, w, prec, ctx), each, max(REL[prec], 1e-15))
