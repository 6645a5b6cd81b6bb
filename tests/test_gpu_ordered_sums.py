"""Smoothing gradients whose sums are taken in a fixed order (GPU): self-pair lists of every order the runs of equal
first spheres can come in, invalid pairs between them, counts around 32 and 64, spheres that are not sorted by link.

Reference and tolerance: as for the other shapes of the kernel, torch.autograd of a float64 restatement; a distance is
off by at most 1.5e-6 m, so with beta = 50 each pair's term is off by at most 1e-4 of itself."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from prrtc_b200 import scenes
from prrtc_b200.context import build_collision_context

pytestmark = pytest.mark.gpu


def _pairs(form: str, pairs: np.ndarray) -> np.ndarray:
    rng = np.random.default_rng(7)
    if form == "reversed":
        return pairs[::-1]
    if form == "shuffled":
        return pairs[rng.permutation(len(pairs))]
    if form == "one_first_sphere":  # runs longer than 32, and every second sphere after its pairs
        return pairs[np.lexsort((pairs[:, 1], pairs[:, 0]))]
    if form == "one_second_sphere":
        return pairs[np.lexsort((pairs[:, 0], pairs[:, 1]))]
    if form == "swapped":
        return pairs[:, ::-1]
    if form == "repeated":
        return np.repeat(pairs[::5], 3, 0)
    if form == "interleaved":  # one first sphere in several runs of 32 pairs
        return pairs.reshape(-1, 32, 2)[:, np.argsort(np.arange(32) % 4, kind="stable")].reshape(-1, 2)
    if form == "invalid":
        out = np.insert(pairs, np.arange(0, len(pairs), 7), -1, axis=0)
        out[3::50, 1] = 10**6
        return out
    if form.startswith("first_"):
        return pairs[:int(form[6:])]
    return pairs


@pytest.mark.parametrize("form", ["by_link", "reversed", "shuffled", "one_first_sphere", "one_second_sphere", "swapped",
                                  "repeated", "interleaved", "invalid", "first_1", "first_31", "first_33", "first_64",
                                  "first_65", "unsorted_spheres"])
def test_pair_lists(cuda, form):
    from oracle.smooth_autodiff import smooth_grad
    from prrtc_b200.smoothing import BatchSmoothContext

    robot = scenes.arm(2)
    base = build_collision_context(robot, None)
    for k in ("coarse_self_pairs", "self_pair_ranges"):
        base[k] = base[k][:0]
    if form == "unsorted_spheres":
        perm = np.random.default_rng(3).permutation(len(base["sphere_link_idx"]))
        for k in ("sphere_link_idx", "sphere_local", "sphere_radius"):
            base[k] = base[k][perm]
        base["self_pairs"] = np.argsort(perm).astype(np.int32)[base["self_pairs"]]
    base["self_pairs"] = np.ascontiguousarray(_pairs(form, base["self_pairs"]))
    S = len(base["sphere_link_idx"])
    worlds = [scenes.tabletop_world(np.random.default_rng(k)) for k in range(2)]
    ctxs = [{**base, **{k: v for k, v in build_collision_context(robot, w).items() if k.startswith("world_")}}
            for w in worlds]
    rng = np.random.default_rng(11)
    x = (rng.uniform(-0.4, 0.4, (2, 1, robot.dim)) + rng.normal(0, 0.05, (2, 9, robot.dim))).astype(np.float32)
    sctx = BatchSmoothContext(ctxs, robot.dim, device=cuda)
    cost, grad = sctx.cost_grad(torch.from_numpy(x).to(cuda))
    again = sctx.cost_grad(torch.from_numpy(x).to(cuda))[1]
    assert torch.equal(grad, again)
    ok = ((base["self_pairs"] >= 0) & (base["self_pairs"] < S)).all(1)
    for p, ctx in enumerate(ctxs):
        c, g = smooth_grad({**ctx, "self_pairs": base["self_pairs"][ok]}, x[p].astype(np.float64), 0.02, 50.0, 1.0)
        assert abs(cost[p].item() - c) <= 1e-4 * abs(c)
        assert np.linalg.norm(grad[p].cpu().numpy().astype(np.float64) - g) <= 5e-4 * np.linalg.norm(g)


@pytest.mark.parametrize("form", ["by_link", "reversed", "shuffled", "swapped", "repeated", "both_ways", "itself", "invalid", "first_1",
                                  "unsorted_spheres"])
def test_pair_lists_of_one_scene(cuda, form):
    """The same lists with one scene for all paths (a lane per waypoint, a pair computed once for each of its spheres):
    lists that repeat a pair, name it both ways or pair a sphere with itself are added up as often as they say."""
    from oracle.smooth_autodiff import smooth_grad
    from prrtc_b200.smoothing import SmoothContext

    robot = scenes.arm(2)
    ctx = build_collision_context(robot, scenes.tabletop_world(np.random.default_rng(3)))
    for k in ("coarse_self_pairs", "self_pair_ranges"):
        ctx[k] = ctx[k][:0]
    if form == "unsorted_spheres":
        perm = np.random.default_rng(3).permutation(len(ctx["sphere_link_idx"]))
        for k in ("sphere_link_idx", "sphere_local", "sphere_radius"):
            ctx[k] = ctx[k][perm]
        ctx["self_pairs"] = np.argsort(perm).astype(np.int32)[ctx["self_pairs"]]
    pairs = ctx["self_pairs"]
    if form == "both_ways":
        pairs = np.concatenate([pairs[:40], pairs[20:60, ::-1], pairs[:3]])
    elif form == "itself":
        pairs = np.insert(pairs, np.arange(0, 100, 9), np.arange(0, 100, 9)[:, None] % 50, axis=0)
    else:
        pairs = _pairs(form, pairs)
    ctx["self_pairs"] = np.ascontiguousarray(pairs)
    rng = np.random.default_rng(11)
    x = (rng.uniform(-0.4, 0.4, (3, 1, robot.dim)) + rng.normal(0, 0.05, (3, 9, robot.dim))).astype(np.float32)
    sctx = SmoothContext(ctx, robot.dim, device=cuda)
    xd = torch.from_numpy(x).to(cuda)
    cost, grad = sctx.cost_grad(xd)
    assert torch.equal(grad, sctx.cost_grad(xd)[1])
    ok = ((pairs >= 0) & (pairs < len(ctx["sphere_link_idx"]))).all(1) & (pairs[:, 0] != pairs[:, 1])
    # a sphere paired with itself: no gradient, and a cost that is added by hand (distance -2 r)
    r = ctx["sphere_radius"][pairs[(pairs[:, 0] == pairs[:, 1]) & (pairs[:, 0] >= 0), 0]].astype(np.float64)
    alone = 9 * float(np.logaddexp(0.0, 50.0 * (0.02 + 2 * r)).sum()) / 50.0
    for p in range(3):
        c, g = smooth_grad({**ctx, "self_pairs": pairs[ok]}, x[p].astype(np.float64), 0.02, 50.0, 1.0)
        assert abs(cost[p].item() - c - alone) <= 1e-4 * abs(c + alone)
        assert np.linalg.norm(grad[p].cpu().numpy().astype(np.float64) - g) <= 5e-4 * np.linalg.norm(g)
