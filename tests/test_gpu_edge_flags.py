"""Edges whose waypoints share a flag (GPU): an edge is free when none of its waypoints is in collision, whatever the order
in which they are tested.  Granularities around a warp and past it, with and without a cloud, colliding edges among
free ones."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from prrtc_b200 import scenes
from prrtc_b200.context import build_collision_context

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cloud", [False, True])
@pytest.mark.parametrize("n,G", [(1, 2), (5, 33), (3, 100), (40, 31), (700, 8), (3000, 3)])
def test_edges_equal_their_waypoints(cuda, n, G, cloud):
    from prrtc_b200 import PointCloud, PointCloudChecker
    from prrtc_b200.collision import CollisionChecker

    robot = scenes.arm(0)
    world, pts = scenes.pointcloud_world(np.random.default_rng(1), 2000)
    ctx = build_collision_context(robot, world)
    rng = np.random.default_rng(n + G)
    a = rng.uniform(robot.lower, robot.upper, (n, 1, robot.dim))
    e = (a + rng.normal(0, 0.1, (n, 1, robot.dim)) * np.linspace(0, 1, G)[None, :, None]).astype(np.float32)
    pc = PointCloud(pts if cloud else np.zeros((0, 3), np.float32), 0.01) if cloud else None
    got = PointCloudChecker(ctx, robot.dim).check_edges_collision_free(e, None, pc, 0.01).cpu().numpy().astype(bool)
    if cloud:  # a waypoint at a time: edges of one
        hit = ~PointCloudChecker(ctx, robot.dim).check_edges_collision_free(
            e.reshape(-1, 1, robot.dim), None, pc, 0.01).cpu().numpy().astype(bool)
    else:
        hit = CollisionChecker(ctx, robot.dim, device=cuda).check(torch.from_numpy(e.reshape(-1, robot.dim))).cpu().numpy() != 0
    assert np.array_equal(got, ~hit.reshape(n, G).any(1))
