"""Smoothing cost and gradient at the edges of the kernel's shapes (GPU): waypoints around a warp, odd and absent
spheres, no self pairs, robots from 2 to 18 joints, one world or one per path, pairs near, far and beyond the tail.

Reference: torch.autograd of a float64 restatement.  A distance is off by at most 1.5e-6 m (float32 frames and a
reciprocal square root of 2 ulp), so with beta = 50 each pair's term is off by at most 1e-4 of itself.
"""
from __future__ import annotations

import numpy as np
import pytest
import torch

from prrtc_b200 import scenes
from prrtc_b200.context import build_collision_context

pytestmark = pytest.mark.gpu


def _paths(robot, P, W, seed):
    rng = np.random.default_rng(seed)
    a, b = rng.uniform(-1.5, 1.5, (2, P, 1, robot.dim))
    t = np.linspace(0.0, 1.0, W)[None, :, None]
    return (a + t * (b - a) + rng.normal(0, 0.02, (P, W, robot.dim))).astype(np.float32)


def _check(cost, grad, ctxs, w, w_len):
    from oracle.smooth_autodiff import smooth_grad

    for p, ctx in enumerate(ctxs):
        c, g = smooth_grad(ctx, w[p].astype(np.float64), 0.02, 50.0, w_len)
        assert abs(cost[p].item() - c) <= 1e-4 * abs(c), (p, cost[p].item(), c)
        got = grad[p].cpu().numpy().astype(np.float64)
        assert np.linalg.norm(got - g) <= 5e-4 * np.linalg.norm(g) + 1e-14, p


@pytest.mark.parametrize("P,W", [(1, 1), (3, 2), (2, 31), (3, 33), (1, 65)])
@pytest.mark.parametrize("joints", [2, 7, 9, 16, 18])
def test_shapes(cuda, P, W, joints):
    from prrtc_b200.smoothing import BatchSmoothContext, SmoothContext

    robot = scenes.dual_arm(0) if joints == 18 else scenes.arm(1, joints)
    worlds = [scenes.tabletop_world(np.random.default_rng(k)) for k in range(P)]
    ctxs = [build_collision_context(robot, w) for w in worlds]
    w = _paths(robot, P, W, joints)
    x = torch.from_numpy(w).to(cuda)
    cost, grad = SmoothContext(ctxs[0], robot.dim, device=cuda).cost_grad(x)
    _check(cost, grad, [ctxs[0]] * P, w, 1.0)
    cost, grad = BatchSmoothContext(ctxs, robot.dim, device=cuda).cost_grad(x)
    _check(cost, grad, ctxs, w, 1.0)


@pytest.mark.parametrize("form", ["odd_spheres", "one_sphere", "no_pairs", "unordered_pairs", "near", "apart", "below_tail"])
def test_forms(cuda, form):
    from prrtc_b200.smoothing import SmoothContext

    robot = scenes.arm(2)
    ctx = build_collision_context(robot, scenes.tabletop_world(np.random.default_rng(4)))
    w_len = 0.0 if form in ("apart", "below_tail") else 0.5
    if form in ("odd_spheres", "one_sphere"):
        n = 1 if form == "one_sphere" else 55
        for k in ("sphere_link_idx", "sphere_local", "sphere_radius"):
            ctx[k] = ctx[k][:n]
        keep = (ctx["self_pairs"] < n).all(1)
        ctx["self_pairs"] = ctx["self_pairs"][keep][::3]
    if form in ("no_pairs", "apart", "below_tail"):
        ctx["self_pairs"] = ctx["self_pairs"][:0]
    if form == "unordered_pairs":
        ctx["self_pairs"] = ctx["self_pairs"][np.random.default_rng(5).permutation(len(ctx["self_pairs"]))[:100]]
    for k in ("coarse_self_pairs", "self_pair_ranges"):
        ctx[k] = ctx[k][:0]
    if form == "near":
        ctx["world_spheres"] = np.concatenate([ctx["world_spheres"], np.array([[0.0, 0.0, 0.5, 0.6]], np.float32)])
    if form in ("apart", "below_tail"):
        at = 0.6 if form == "apart" else 1.05  # about 0.4 m and 0.85 m from the nearest link
        for k in list(ctx):
            if k.startswith("world_"):
                ctx[k] = ctx[k][:0]
        ctx["world_spheres"] = np.array([[at, 0.0, 0.5, 0.1], [at, 0.3, 0.5, 0.1]], np.float32)
    w = 0.2 * _paths(robot, 2, 40, 9)
    cost, grad = SmoothContext(ctx, robot.dim, w_len=w_len, device=cuda).cost_grad(torch.from_numpy(w).to(cuda))
    _check(cost, grad, [ctx] * 2, w, w_len)
    if form == "below_tail":
        assert 0.0 < cost.max().item() < 1e-15 and float(grad.abs().max()) < 1e-13


def test_paths_without_a_world(cuda):
    """A context of None is a path without world or self pairs; re-validation with no device named answers on torch's
    default one."""
    from prrtc_b200.smoothing import BatchSmoothContext, SmoothContext, revalidate_batch

    robot = scenes.arm(0)
    ctx = build_collision_context(robot, scenes.tabletop_world(np.random.default_rng(4)))
    empty = {k: v[:0] if k.startswith("world_") or k == "self_pairs" else v for k, v in ctx.items()}
    for k in ("coarse_self_pairs", "self_pair_ranges"):
        empty[k] = empty[k][:0]
    x = torch.from_numpy(_paths(robot, 3, 9, 2)).to(cuda)
    ctxs = [ctx, None, ctx]
    cost, grad = BatchSmoothContext(ctxs, robot.dim, device=cuda).cost_grad(x)
    for p, c in enumerate((ctx, empty, ctx)):
        c1, g1 = SmoothContext(c, robot.dim, device=cuda).cost_grad(x[p:p + 1], ordered=True)
        assert torch.equal(grad[p], g1[0])
        assert abs(cost[p].item() - c1.item()) <= 2e-6 * abs(c1.item())  # 9 waypoints' costs in any order
    want = revalidate_batch(x, ctxs, 0.02, cuda)
    got = revalidate_batch(x, ctxs, 0.02, None)
    assert got.device == torch.empty(0).device and torch.equal(got, want.cpu()) and bool(want[1])
    assert torch.equal(revalidate_batch(x, [ctx] * 3, 0.02, None), revalidate_batch(x, [ctx] * 3, 0.02, cuda).cpu())


@pytest.mark.parametrize("bad", [np.nan, np.inf])
@pytest.mark.parametrize("scene", ["spheres", "capsules", "boxes", "halfspaces", "self_pairs", "all"])
def test_a_waypoint_that_is_not_a_number(cuda, scene, bad):
    """A path of one waypoint with a coordinate that is not a number (no length term carries it): its cost and every
    gradient entry that depends on it are not numbers either, and the paths beside it keep their values."""
    from prrtc_b200.smoothing import SmoothContext

    robot = scenes.arm(2)
    ctx = build_collision_context(robot, scenes.tabletop_world(np.random.default_rng(4)))
    for k in ("world_spheres", "world_capsules", "world_boxes", "world_halfspaces", "self_pairs"):
        if scene != "all" and not k.endswith(scene):
            ctx[k] = ctx[k][:0]
    for k in ("coarse_self_pairs", "self_pair_ranges"):
        ctx[k] = ctx[k][:0]
    sctx = SmoothContext(ctx, robot.dim, device=cuda)
    x = torch.from_numpy(_paths(robot, 3, 1, 6)).to(cuda)
    want_cost, want_grad = sctx.cost_grad(x)
    x[1, 0, 1] = bad
    cost, grad = sctx.cost_grad(x)
    assert torch.isnan(cost).tolist() == [False, True, False]
    assert torch.equal(torch.isnan(grad), torch.isnan(sctx.cost_grad(x, ordered=True)[1])) and bool(torch.isnan(grad[1]).any())
    for p in (0, 2):  # neighbouring lanes may take the full softplus with it: a term's rounding, at most 1e-6 of it
        assert torch.allclose(cost[p], want_cost[p], rtol=1e-5, atol=0.0)
        assert torch.allclose(grad[p], want_grad[p], rtol=1e-5, atol=1e-5 * float(want_grad[p].abs().max()))


@pytest.mark.parametrize("joints,P,W", [(7, 1, 64), (7, 14, 33), (7, 97, 33), (7, 194, 33), (7, 427, 33), (18, 3, 40), (18, 90, 40)])
def test_gradients_are_the_same_bits_in_every_run(cuda, joints, P, W):
    """From a few waypoints, shared by eight CTAs, to more than the GPU holds at once: five calls, the same gradient,
    and the one of the kernel with a warp per waypoint within the two kernels' bounds (each 5e-4 of the path's)."""
    from prrtc_b200.smoothing import SmoothContext

    robot = scenes.dual_arm(0) if joints == 18 else scenes.arm(1, joints)
    world = scenes.large_world(np.random.default_rng(3)) if joints == 18 else scenes.tabletop_world(np.random.default_rng(3))
    sctx = SmoothContext(build_collision_context(robot, world), robot.dim, device=cuda)
    x = torch.from_numpy(_paths(robot, P, W, 5)).to(cuda)
    grads = [sctx.cost_grad(x)[1].clone() for _ in range(5)]
    assert all(torch.equal(g, grads[0]) for g in grads[1:])
    want = sctx.cost_grad(x, ordered=True)[1]
    off = torch.linalg.norm((grads[0] - want).reshape(P, -1), dim=1)
    assert bool((off <= 1e-3 * torch.linalg.norm(want.reshape(P, -1), dim=1)).all())


@pytest.mark.parametrize("spheres", [1200, 1764, 1790, 1795])
def test_robots_of_many_spheres(cuda, spheres):
    """Robots whose sphere tables fill shared memory: scenes that are not staged, up to the largest robot that four
    waypoints per CTA took before their sums had a row of their own (1,795 spheres with 7 joints)."""
    from prrtc_b200.smoothing import BatchSmoothContext, SmoothContext

    robot = scenes.arm(2)
    ctx = build_collision_context(robot, scenes.spheres_world(np.random.default_rng(4), 3))
    rng = np.random.default_rng(8)
    pick = rng.integers(0, len(ctx["sphere_link_idx"]), spheres)
    for k in ("sphere_link_idx", "sphere_local", "sphere_radius"):
        ctx[k] = ctx[k][pick]
    ctx["sphere_local"] = (ctx["sphere_local"] + rng.uniform(-0.01, 0.01, (spheres, 3))).astype(np.float32)
    ctx["self_pairs"] = ctx["self_pairs"][:7]
    for k in ("coarse_self_pairs", "self_pair_ranges"):
        ctx[k] = ctx[k][:0]
    w = _paths(robot, 2, 3, 9)
    x = torch.from_numpy(w).to(cuda)
    for got in (SmoothContext(ctx, robot.dim, device=cuda).cost_grad(x), BatchSmoothContext([ctx] * 2, robot.dim, device=cuda).cost_grad(x)):
        _check(*got, [ctx] * 2, w, 1.0)
