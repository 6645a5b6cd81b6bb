"""Smoothing with the sums in the batched entry's order, and the batched descent (GPU).

Values against torch.autograd of a float64 restatement with the bounds of the other shapes of the kernel (a distance is
off by at most 1.5e-6 m, so with beta = 50 a pair's term by at most 1e-4 of itself); the descent against the tensor
expression that it stands for, whose operations and order it takes over: the same bits."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from prrtc_b200 import scenes
from prrtc_b200.context import build_collision_context, with_world
from test_gpu_fk_shapes import _tables
from test_gpu_smoothing_shapes import _check, _paths

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("P,W", [(1, 1), (3, 2), (3, 33)])
def test_ordered_sums_of_one_scene(cuda, P, W):
    """Eight waypoints per CTA, which span paths: a path's gradient is the batched entry's, whatever is beside it."""
    from prrtc_b200.smoothing import BatchSmoothContext, SmoothContext

    robot = scenes.arm(1)
    ctx = build_collision_context(robot, scenes.tabletop_world(np.random.default_rng(2)))
    w = _paths(robot, P, W, 3)
    x = torch.from_numpy(w).to(cuda)
    sctx = SmoothContext(ctx, robot.dim, device=cuda)
    cost, grad = sctx.cost_grad(x, ordered=True)
    _check(cost, grad, [ctx] * P, w, 1.0)
    assert torch.equal(grad, BatchSmoothContext([ctx] * P, robot.dim, device=cuda).cost_grad(x)[1])
    for p in range(P):
        assert torch.equal(sctx.cost_grad(x[p:p + 1], ordered=True)[1][0], grad[p])


@pytest.mark.parametrize("joints", [33, 64])
def test_more_joints_than_lanes(cuda, joints):
    from prrtc_b200.smoothing import BatchSmoothContext, SmoothContext

    rng = np.random.default_rng(joints)
    dim = 16
    ctx = {**_tables(joints, dim, joints), "sphere_link_idx": np.arange(joints, dtype=np.int32),
           "sphere_local": rng.uniform(-0.02, 0.02, (joints, 3)).astype(np.float32),
           "sphere_radius": rng.uniform(0.02, 0.04, joints).astype(np.float32),
           "self_pairs": np.array([(i, j) for i in range(joints) for j in range(i + 9, joints, 5)], np.int32)}
    ctx = with_world(ctx, scenes.tabletop_world(np.random.default_rng(2)))
    w = rng.uniform(-1.0, 1.0, (2, 3, dim)).astype(np.float32)
    x = torch.from_numpy(w).to(cuda)
    _check(*SmoothContext(ctx, dim, device=cuda).cost_grad(x), [ctx] * 2, w, 1.0)
    _check(*BatchSmoothContext([ctx] * 2, dim, device=cuda).cost_grad(x), [ctx] * 2, w, 1.0)


@pytest.mark.parametrize("limit", ["numbers", "nan"])
@pytest.mark.parametrize("W", [3, 17])
def test_descent_is_the_tensor_expression(cuda, W, limit):
    """Paths at their limits, one whose gradient is zero and one that is not a number; a limit that is not a number
    spreads to every path with a gradient."""
    from prrtc_b200.smoothing import BatchSmoothContext, projected_steps

    robot = scenes.arm(0)
    base = build_collision_context(robot, None)
    ctxs = [with_world(base, scenes.tabletop_world(np.random.default_rng(k))) for k in range(5)]
    ctxs[3] = {**ctxs[3], **{k: v[:0] for k, v in ctxs[3].items() if k.startswith("world_") or k == "self_pairs"}}
    x = torch.from_numpy(_paths(robot, 5, W, 7)).to(cuda)
    x[3] = x[3, :1]
    x[4, 1, 2] = np.nan
    lo, hi = torch.full((robot.dim,), -0.8, device=cuda), torch.full((robot.dim,), 0.7, device=cuda)
    if limit == "nan":
        hi[5] = np.nan
    sctx = BatchSmoothContext(ctxs, robot.dim, device=cuda)
    got = projected_steps(sctx, x, lo, hi, 4, 0.05)
    want = x.clone()
    mask = torch.ones_like(x)
    mask[:, 0] = mask[:, -1] = 0.0
    for _ in range(4):
        g = torch.where(mask > 0, sctx.cost_grad(want)[1], torch.zeros_like(want))
        gn = torch.linalg.norm(g.reshape(5, -1), dim=1).clamp_min(1e-12)
        want = torch.minimum(torch.maximum(want - 0.05 * g / gn[:, None, None], lo), hi)
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    assert torch.equal(torch.nan_to_num(got), torch.nan_to_num(want))
    if limit == "numbers":
        assert bool((got[:3] == -0.8).any()) and torch.equal(got[3, 0], x[3, 0].clamp(-0.8, 0.7))
