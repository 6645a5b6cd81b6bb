"""Nearest neighbour at the edges of the scan's shapes (GPU): queries around a CTA's share, every block count of
dimensions, rows that start unaligned, sizes around a column of 1024 nodes, ties across CTAs, unwritten (NaN) and
overflowing nodes.  The oracle's sequential scan must be matched bit for bit."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _check(orc, tree, n, q, view=None):
    from prrtc_b200 import prrtc_nearest_neighbor

    dist, idx = prrtc_nearest_neighbor(tree if view is None else view, q, n)
    oi, od = orc.nearest_batch(tree.cpu().numpy(), n, q.cpu().numpy())
    assert np.array_equal(idx.cpu().numpy(), oi)
    want = np.sqrt(od.astype(np.float32))
    assert np.array_equal(dist.cpu().numpy().view(np.uint32), want.view(np.uint32))


@pytest.mark.parametrize("batch", [1, 3, 4, 63, 65, 200])
@pytest.mark.parametrize("dim,N,n", [(1, 1024, 1), (4, 1023, 1023), (5, 1025, 1025), (7, 200004, 199999), (8, 40961, 30000),
                                     (9, 5003, 4097), (13, 3000, 2999), (16, 2048, 2048)])
def test_shapes(cuda, orc, batch, dim, N, n):
    g = torch.Generator(device=cuda).manual_seed(dim * 1000 + batch)
    tree = torch.rand((dim, N), generator=g, device=cuda) * 5.6 - 2.8
    tree[:, n:] = float("nan")
    tree[dim - 1, ::5] = float("nan")  # half-written nodes
    tree[:, 0] = 1.0
    q = torch.rand((batch, dim), generator=g, device=cuda) * 5.6 - 2.8
    _check(orc, tree, n, q)


@pytest.mark.parametrize("N", [60000, 60001])
def test_ties_and_far_nodes(cuda, orc, N):
    """The same node over and over: the lowest index wins whichever CTA finds it first.  Distances that overflow and
    trees without a node give index 0 at infinity."""
    from prrtc_b200 import prrtc_nearest_neighbor

    rng = np.random.default_rng(N)
    base = rng.uniform(-1, 1, (7, 41)).astype(np.float32)
    tree = torch.from_numpy(np.tile(base, (1, N // 41 + 1))[:, :N].copy()).to(cuda)
    q = torch.from_numpy(np.concatenate([base[:, ::-1].T, rng.uniform(-1, 1, (30, 7)).astype(np.float32)]).copy()).to(cuda)
    _check(orc, tree, N, q)
    for fill in (1e30, float("nan"), float("inf")):
        dist, idx = prrtc_nearest_neighbor(torch.full((7, N), fill, device=cuda), q, N)
        assert bool((idx == 0).all()) and bool(torch.isinf(dist).all())
