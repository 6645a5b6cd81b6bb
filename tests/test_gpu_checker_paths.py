"""Scene packing and the batched checker's paths on scenes at the edges of their ranges (GPU).

Every form of a scene is checked by the default path and by the full sweep, which tests every pair; both must
give the verdicts of the plain scene that the form restates.
"""
from __future__ import annotations

import numpy as np
import pytest

from prrtc_b200 import scenes
from prrtc_b200.context import build_collision_context

pytestmark = pytest.mark.gpu

CHECKERS = ["binary", "differentiable", "binary_coarse", "binary_coarse_coop"]


def _verdicts(ctx, robot, mode, q, cuda):
    from prrtc_b200.collision import CollisionChecker

    chk = CollisionChecker(ctx, robot.dim, CHECKERS[mode], 0.02, device=cuda)
    early = chk.check(q).cpu().numpy()
    full = chk.check(q, full_sweep=True).cpu().numpy()
    assert np.array_equal(early, full)
    return early


def _repeat_pairs(ctx, times):
    out = dict(ctx)
    P = len(ctx["self_pairs"])
    out["self_pairs"] = np.tile(ctx["self_pairs"], (times, 1))
    out["coarse_self_pairs"] = np.tile(ctx["coarse_self_pairs"], (times, 1))
    out["self_pair_ranges"] = np.concatenate([ctx["self_pair_ranges"] + P * k for k in range(times)]).astype(np.int32)
    return out


@pytest.mark.parametrize("mode", [0, 1, 2, 3])
@pytest.mark.parametrize("form", ["one_tile", "two_tiles", "unordered_range", "overlapping_ranges", "gaps"])
def test_self_pair_items(cuda, mode, form):
    """Coarse pairs at and past one packing tile (512), ranges that are not blocks, ranges that overlap (more
    items than the list holds: the flat pair list is used) and ranges that leave pairs out."""
    robot = scenes.arm(3)
    ctx = build_collision_context(robot, scenes.spheres_world(np.random.default_rng(5), 16))
    q = np.random.default_rng(6).uniform(robot.lower, robot.upper, (400, robot.dim)).astype(np.float32)
    want = _verdicts(ctx, robot, mode, q, cuda)
    got = dict(ctx)
    if form == "one_tile":
        got = _repeat_pairs(ctx, 34)  # 510 coarse pairs
    elif form == "two_tiles":
        got = _repeat_pairs(ctx, 35)  # 525
    elif form == "unordered_range":
        p = ctx["self_pairs"].copy()
        p[70:90] = p[70:90][::-1]
        got["self_pairs"] = p
    elif form == "overlapping_ranges":
        P, Q = len(ctx["self_pairs"]), len(ctx["self_pair_ranges"])
        got["self_pair_ranges"] = np.tile(np.array([[0, P]], np.int32), (Q, 1))
        want = _verdicts(ctx, robot, 0 if mode > 1 else mode, q, cuda)  # the flat sweep of every pair
    else:
        # the ranges of every second coarse pair: a gated checker tests those pairs, a flat one all
        keep = np.arange(0, len(ctx["self_pair_ranges"]), 2)
        got["coarse_self_pairs"] = ctx["coarse_self_pairs"][keep]
        got["self_pair_ranges"] = ctx["self_pair_ranges"][keep]
        if mode > 1:
            rows = np.concatenate([np.arange(a, b) for a, b in got["self_pair_ranges"]])
            part = dict(ctx, self_pairs=ctx["self_pairs"][rows])
            part["coarse_self_pairs"] = part["self_pair_ranges"] = np.zeros((0, 2), np.int32)
            want = _verdicts(part, robot, 0, q, cuda)
    assert np.array_equal(_verdicts(got, robot, mode, q, cuda), want)
