"""Nearest neighbour of batches on large trees (GPU), where the tensor cores rule nodes out first: node counts around a
warp's 32 nodes and the first scan, batches around a tile of 8 queries, unaligned rows, duplicates and ties, nodes that
come nearer with their index, NaN, infinite, huge and tiny values.  The oracle's sequential scan must be matched bit for
bit."""
from __future__ import annotations

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

CAP = 1 << 19  # 16 queries and 2^23 pairs: the first size that takes the filter


def _check(orc, tree, n, q):
    from prrtc_b200 import prrtc_nearest_neighbor

    dist, idx = prrtc_nearest_neighbor(tree, q, n)
    oi, od = orc.nearest_batch(tree.cpu().numpy(), n, q.cpu().numpy())
    assert np.array_equal(idx.cpu().numpy(), np.maximum(oi, 0))  # no node in reach: index 0 at infinity
    assert np.array_equal(dist.cpu().numpy().view(np.uint32), np.sqrt(od.astype(np.float32)).view(np.uint32))


@pytest.mark.parametrize("dim", [1, 7, 8, 14, 15, 16])
@pytest.mark.parametrize("batch,N,n", [(16, CAP, CAP), (17, CAP + 1, CAP - 31), (32, CAP + 4, 8193), (33, CAP + 2, 8192),
                                       (64, CAP + 12, CAP + 11), (65, CAP, 100001), (15, CAP, CAP)])
def test_shapes(cuda, orc, dim, batch, N, n):
    g = torch.Generator(device=cuda).manual_seed(dim * 100 + batch)
    tree = torch.rand((dim, N), generator=g, device=cuda) * 5.6 - 2.8
    tree[:, n:] = float("nan")
    tree[dim - 1, ::1001] = float("nan")  # half-written nodes
    tree[:, 0] = 1.0
    q = torch.rand((batch, dim), generator=g, device=cuda) * 5.6 - 2.8
    _check(orc, tree, n, q)


@pytest.mark.parametrize("form", ["same", "grid", "on_nodes", "nearing", "far_origin", "tiny", "huge", "overflow", "inf_nodes",
                                  "nan_nodes", "odd_queries"])
def test_values(cuda, orc, form):
    dim, n, batch = 7, CAP - 5, 20
    rng = np.random.default_rng(3)
    tree = rng.uniform(-2.8, 2.8, (dim, CAP)).astype(np.float32)
    q = rng.uniform(-2.8, 2.8, (batch, dim)).astype(np.float32)
    if form == "same":  # every node a tie
        tree[:] = 0.3
    elif form == "grid":
        tree, q = np.round(tree).astype(np.float32), np.round(q).astype(np.float32)
    elif form == "on_nodes":
        q = np.ascontiguousarray(tree[:, rng.integers(0, n, batch)].T)
    elif form == "nearing":  # every node nearer than those before it
        tree = (q[:1].T + np.linspace(2.0, 0.01, CAP)[None] * np.ones((dim, 1))).astype(np.float32)
    elif form == "far_origin":  # distances far below the norms' rounding
        tree, q = tree * np.float32(1e-3) + np.float32(1000), q * np.float32(1e-3) + np.float32(1000)
    elif form == "tiny":
        tree, q = tree * np.float32(1e-21), q * np.float32(1e-21)
    elif form == "huge":
        tree, q = tree * np.float32(1e18), q * np.float32(1e18)
    elif form == "overflow":
        tree, q = tree * np.float32(1e19), q * np.float32(5e18)
    elif form == "inf_nodes":
        tree[2, ::3] = np.inf
        tree[3, 1::3] = -np.inf
    elif form == "nan_nodes":
        tree[5, np.arange(CAP) % 16 != 3] = np.nan
    elif form == "odd_queries":
        q[0, 0], q[1, 1], q[2] = np.nan, np.inf, 3e38
    _check(orc, torch.from_numpy(tree).to(cuda), n, torch.from_numpy(np.ascontiguousarray(q)).to(cuda))
