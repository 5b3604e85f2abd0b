"""GPU: the MLP's 128-row tiles at their edges.  A row's output does not depend
on the tile it falls in, so a forward pass over a part of the rows gives the
same bits; gradients of batches of less than a tile, one row more than a tile
and several are compared with the numpy restatement."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import mlp_oracle as MO

pytestmark = pytest.mark.gpu

REL = 2e-2   # bf16 activations, as in the other comparisons with this restatement


def rel(a, b):
    return float(np.linalg.norm(np.asarray(a, np.float64) - b) / max(np.linalg.norm(b), 1e-30))


def problem(ctx, n):
    import torch
    from phylocaml_gb300 import mlp
    rng = np.random.default_rng(n)
    X = rng.normal(size=(n, 64)).astype(np.float32) * rng.uniform(0.5, 3, 64).astype(np.float32)
    t = (np.tanh(X[:, 0]) - 0.3 * X[:, 1] * X[:, 2]).astype(np.float32)
    net = mlp.MLP(seed=5, max_batch=700, ctx=ctx)
    net.fit_norm(torch.from_numpy(rng.normal(size=(400, 64)).astype(np.float32)).cuda())
    return net, X, t


def test_forward_rows_do_not_depend_on_their_tile(ctx):
    import torch
    net, X, _ = problem(ctx, 40001)   # more tiles than two per SM
    mu, inv = net.norm()
    Xd = torch.from_numpy(X).cuda()
    whole = net.forward(Xd).cpu().numpy()
    assert rel(whole[:2000], MO.forward(net.params(), mu, inv, X[:2000])[0]) < REL
    for n in (1, 2, 127, 128, 129, 255, 256, 257, 1000):
        for at in (0, 64, 39000):
            got = net.forward(Xd[at:at + n].contiguous()).cpu().numpy()
            assert np.array_equal(got, whole[at:at + n]), (n, at)
    net.close()


@pytest.mark.parametrize("n", [1, 127, 128, 129, 512, 700])
@pytest.mark.parametrize("weighted", [False, True])
def test_gradients_at_tile_edges(ctx, n, weighted):
    import torch
    from phylocaml_gb300 import mlp
    net, X, t = problem(ctx, n)
    mu, inv = net.norm()
    sw = np.random.default_rng(3).uniform(0.5, 2, n).astype(np.float32) if weighted else None
    dev = [None if v is None else torch.from_numpy(v).cuda() for v in (X, t, sw)]
    g, loss = net.grads(*dev)
    exp_loss, exp_g = MO.loss_and_grads(net.params(), mu, inv, X, t, sw)
    assert abs(loss - exp_loss) <= 1e-2 * exp_loss + 1e-6
    for name, (o, s) in mlp.param_slices().items():
        k = int(np.prod(s))
        assert rel(g[o:o + k], exp_g[o:o + k]) < REL, name
    net.close()
