"""GPU: a tree that is new to a context is refused while the context's stream
is captured into a CUDA graph -- its schedule would be recorded instead of
copied, and every later call on that tree would trust what is not there -- and
nothing is kept of the refused call.  A tree the context knows is recorded and
replays."""
from __future__ import annotations

import numpy as np
import pytest

from phylocaml_gb300 import _native, costmatrix, fitch, likelihood, mlmodel as M, synth, tree as T

pytestmark = pytest.mark.gpu

SITES = 1000


def calls(ctx, rng):
    """(name, run(tree, result), result) of every device call that keeps
    something of a tree; the buffers fit the larger tree."""
    import torch
    dev = torch.device("cuda:0")
    n = 40
    out = []

    def packed(lanes, states):
        codes = (1 << rng.integers(0, states, (n, SITES))).astype({4: np.uint8, 8: np.uint8, 32: np.uint32}[lanes])
        raw = codes[:, 0::2] | codes[:, 1::2] << 4 if lanes == 4 else codes
        raw = np.ascontiguousarray(raw).view(np.uint8)
        words = np.zeros((n, (raw.shape[1] + 15) // 16 * 16), np.uint8)
        words[:, :raw.shape[1]] = raw
        return torch.from_numpy(words.view(np.int32)).to(dev)

    tensor = lambda *shape, t=torch.int32: torch.zeros(shape, dtype=t, device=dev)   # noqa: E731
    for lanes in (4, 64):
        tips = torch.from_numpy(rng.integers(1, 1 << 31, (n, 2000)).astype(np.int32)).to(dev) if lanes == 64 \
            else packed(4, 4)
        sets, cost = tensor(n - 1, tips.shape[1]), tensor(SITES)
        out.append((f"fitch {lanes}", lambda tr, total, tips=tips, sets=sets, cost=cost, lanes=lanes:
                    fitch.fitch_tree_dev(tr, tips, tips.shape[1], SITES, lanes, None, sets, cost, total, ctx),
                    tensor(1, t=torch.int64)))
    for states, lanes in ((4, 4), (20, 32)):
        c = rng.integers(1, 4, (states, states)).astype(np.int32)
        np.fill_diagonal(c, 0)
        m = costmatrix.CostMatrix(c, "general")
        tips = packed(lanes, states)
        sets, cost = tensor(n - 1, tips.shape[1]), tensor(SITES)
        out.append((f"tcm {states}", lambda tr, total, m=m, tips=tips, sets=sets, cost=cost:
                    m.tree_cost_dev(tr, tips, tips.shape[1], SITES, None, sets, cost, total, ctx),
                    tensor(1, t=torch.int64)))
    model = M.create(synth.random_gtr_spec(rng, 0.5, 4), ctx)
    codes = torch.from_numpy(rng.integers(1, 16, (n, 1008)).astype(np.uint8)).to(dev)
    out.append(("prune", lambda tr, lnl: likelihood.tree_lnl_dev(tr, model, codes, 1008, SITES, synth.dna_code_table(),
                                                                 None, lnl, 48, None, ctx),
                tensor(1, t=torch.float64)))
    return out


def test_new_tree_under_capture(native_lib):
    import torch
    rng = np.random.default_rng(5)
    large, small = T.yule(40, rng, 0.1), T.yule(24, rng, 0.1)
    stream = torch.cuda.Stream()
    with _native.Context(0) as ctx, _native.Context(0) as other:
        ctx.set_stream(stream.cuda_stream)
        want = {}
        for name, run, result in calls(other, np.random.default_rng(7)):
            torch.cuda.synchronize()
            run(small, result)
            other.synchronize()
            torch.cuda.synchronize()
            want[name] = result.item()
        for name, run, result in calls(ctx, np.random.default_rng(7)):
            torch.cuda.synchronize()
            with torch.cuda.stream(stream):
                run(large, result)              # the context's buffers exist
            ctx.synchronize()
            graph = torch.cuda.CUDAGraph()
            with torch.cuda.graph(graph, stream=stream):
                with pytest.raises(_native.NativeError, match="captured"):
                    run(small, result)
                torch.zeros(1, device="cuda:0")
            del graph
            with torch.cuda.stream(stream):
                run(small, result)              # uploads the tree: nothing was kept
            ctx.synchronize()
            assert result.item() == want[name], name
            if name.startswith("fitch"):        # no per-call parameters: a known tree replays
                graph = torch.cuda.CUDAGraph()
                with torch.cuda.graph(graph, stream=stream):
                    run(small, result)
                result.zero_()
                torch.cuda.synchronize()
                graph.replay()
                torch.cuda.synchronize()
                assert result.item() == want[name], name
        ctx.set_stream(None)
