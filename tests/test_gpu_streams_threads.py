"""Objects used on another stream than the one they were made on, and calls from several host threads (GPU)."""
from __future__ import annotations

import threading

import numpy as np
import pytest
import torch

from prrtc_b200 import scenes
from prrtc_b200.context import build_collision_context, with_world

pytestmark = pytest.mark.gpu


def _paths(robot, P, W, seed, device):
    q = np.random.default_rng(seed).uniform(-1.0, 1.0, (P, W, robot.dim)).astype(np.float32)
    return torch.from_numpy(q).to(device)


def test_batch_smoothing_context_on_another_stream(cuda):
    """Built on a stream with work in front, evaluated at once on another stream: the tables have to be there."""
    from prrtc_b200.smoothing import BatchSmoothContext

    robot = scenes.arm(0)
    base = build_collision_context(robot, None)
    ctxs = [with_world(base, scenes.tabletop_world(np.random.default_rng(k))) for k in range(5)]
    x = _paths(robot, 5, 17, 3, cuda)
    cost, grad = BatchSmoothContext(ctxs, robot.dim, device=cuda).cost_grad(x)
    torch.cuda.synchronize()
    one, other = torch.cuda.Stream(cuda), torch.cuda.Stream(cuda)
    with torch.cuda.stream(one):
        torch.cuda._sleep(100_000_000)  # about 50 ms
        sctx = BatchSmoothContext(ctxs, robot.dim, device=cuda)
    with torch.cuda.stream(other):
        got_cost, got_grad = sctx.cost_grad(x)
    torch.cuda.synchronize()
    # the sums of a gradient have one order; a path's cost is added up over its waypoints in any order (17 terms of one
    # sign: 16 roundings of 2^-24 each)
    assert torch.equal(got_grad, grad)
    assert torch.allclose(got_cost, cost, rtol=2e-6, atol=0.0)
