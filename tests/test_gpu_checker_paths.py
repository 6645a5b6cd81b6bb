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


def _odd_scene(form, rng):
    """A scene at the edge of what the culled edge check takes (or past it), and its robot."""
    robot = scenes.arm(0)
    ctx = build_collision_context(robot, scenes.uneven_world(rng) if form == "plain" else scenes.tabletop_world(rng))
    if form == "many":  # more primitives around every link than a link's list holds (256)
        s = scenes.spheres_world(rng, 700)["world_spheres"]
        s[:, 3] = 0.01
        ctx["world_spheres"] = s
    elif form == "far_sphere":  # a link that reaches past the culled range touches every primitive: full lists
        ctx["sphere_local"] = ctx["sphere_local"].copy()
        ctx["sphere_local"][20] = (0.0, 0.0, 40.0)
    elif form == "uncovered":  # groups that do not cover the first sphere
        ctx["fine_link_offsets"] = ctx["fine_link_offsets"].copy()
        ctx["fine_link_offsets"][0] = 1
    elif form == "mixed_frames":  # a sphere listed in another link's group
        ctx["sphere_link_idx"] = ctx["sphere_link_idx"].copy()
        ctx["sphere_link_idx"][17] = 0
    elif form == "small_coarse":  # coarse spheres that do not enclose their fine spheres (flat checkers ignore them)
        ctx["coarse_sphere_radius"] = ctx["coarse_sphere_radius"] * 0.1
    elif form == "long_normal":
        ctx["world_halfspaces"] = np.array([[0, 0, 3.0, 0, 0, 0.02]], np.float32)
    elif form == "sheared_boxes":
        ctx["world_boxes"] = ctx["world_boxes"].copy()
        ctx["world_boxes"][:, 3:12] *= 1.5
        ctx["world_boxes"][::2, 3] += 0.4
    elif form == "negative_radii":
        ctx["world_spheres"] = ctx["world_spheres"].copy()
        ctx["world_spheres"][::3, 3] *= -1
        ctx["world_capsules"] = ctx["world_capsules"].copy()
        ctx["world_capsules"][0, 6] *= -1
    elif form == "nan_and_far":
        ctx["world_spheres"] = np.concatenate([ctx["world_spheres"], np.array(
            [[np.nan, 0, 0, 0.1], [3e5, -2e5, 1e5, 0.2], [np.inf, 0, 0, 0.1]], np.float32)])
        ctx["world_capsules"] = np.concatenate([ctx["world_capsules"], ctx["world_capsules"][:1]])
        ctx["world_capsules"][-1, 3:6] = ctx["world_capsules"][-1, :3] + 1e-25  # no length
    return robot, ctx


FORMS = ["plain", "many", "far_sphere", "uncovered", "mixed_frames", "small_coarse", "long_normal", "sheared_boxes",
         "negative_radii", "nan_and_far"]
COARSE = ("coarse_sphere_link_idx", "coarse_sphere_local", "coarse_sphere_radius", "fine_link_offsets",
          "coarse_self_pairs", "self_pair_ranges")


@pytest.mark.parametrize("checker", ["binary", "differentiable"])
@pytest.mark.parametrize("form", FORMS)
def test_culled_plans_equal_general_plans(cuda, form, checker):
    """One explorer per problem: the same scene with its coarse model (culled edge checks) and without it (the
    general checker) must give the same plans, bit for bit -- wide, ordinary and plain launches."""
    from prrtc_b200 import prrtc_plan_batch

    robot, ctx = _odd_scene(form, np.random.default_rng(11))
    bare = {k: v for k, v in ctx.items() if k not in COARSE}
    B = 6
    # starts and goals need not be free: a plan that fails has to fail alike
    q = np.random.default_rng(12).uniform(-1.2, 1.2, (2, B, robot.dim)).astype(np.float32)
    kw = dict(max_iterations=60, num_new_samples=1, max_nodes=2048, min_vals=robot.lower, max_vals=robot.upper,
              collision_checker=checker, edge_resolution=0.02, tail_explorers=False)

    def plan(c, launch, threads):
        return prrtc_plan_batch(q[0], q[1][:, None], collision_context=[c] * B, launch=launch,
                                threads_per_explorer=threads, waypoint_chunk=16, **kw)

    want = plan(bare, "persistent", 128)
    for launch, threads in (("persistent", 0), ("per_problem", 64), ("per_problem", 256)):
        for a, b in zip(plan(ctx, launch, threads), want):
            assert (a.solved, a.tree_a_size, a.tree_b_size, a.iterations) == (
                b.solved, b.tree_a_size, b.tree_b_size, b.iterations), (launch, threads)
            for x, y in ((a.tree_a_configs, b.tree_a_configs), (a.tree_b_configs, b.tree_b_configs)):
                assert np.array_equal(x.cpu().numpy().view(np.uint32), y.cpu().numpy().view(np.uint32)), (launch, threads)


@pytest.mark.parametrize("n_joints", [2, 8, 9, 16])
def test_culled_plans_across_joint_counts(cuda, n_joints):
    """Joint counts at the edges of a waypoint's lane segment (8, 16, 32), large trees in a scan's second round."""
    from prrtc_b200 import prrtc_plan_batch

    robot = scenes.arm(1, n_joints)
    ctx = build_collision_context(robot, scenes.dense_world(np.random.default_rng(2)))
    bare = {k: v for k, v in ctx.items() if k not in COARSE}
    q = np.random.default_rng(3).uniform(-1.0, 1.0, (2, 3, robot.dim)).astype(np.float32)
    kw = dict(max_iterations=300, num_new_samples=1, max_nodes=1025, min_vals=robot.lower, max_vals=robot.upper,
              step_size=0.1, edge_resolution=0.013, tail_explorers=False, dynamic_domain=False)
    a = prrtc_plan_batch(q[0], q[1][:, None], collision_context=ctx, **kw)
    b = prrtc_plan_batch(q[0], q[1][:, None], collision_context=bare, **kw)
    for x, y in zip(a, b):
        assert (x.solved, x.tree_a_size, x.tree_b_size, x.iterations) == (y.solved, y.tree_a_size, y.tree_b_size,
                                                                          y.iterations)
        assert np.array_equal(x.tree_a_configs.cpu().numpy().view(np.uint32), y.tree_a_configs.cpu().numpy().view(np.uint32))


@pytest.mark.parametrize("checker", ["binary", "binary_coarse_coop"])
@pytest.mark.parametrize("cell,r_env", [(0.1, 0.01), (0.1, 0.0), (0.02, 0.005), (0.013, 0.02), (1.0, 0.05)])
def test_cloud_batches_equal_general_checker(cuda, cell, r_env, checker):
    """Point clouds: cells from smaller than the spheres (a box of more than 512 cells is a hit) to larger than the
    cloud, points on the far side of the coordinate limit, edge counts around a warp; and plans with a cloud."""
    from prrtc_b200 import PointCloud, PointCloudChecker, prrtc_plan_batch

    robot = scenes.arm(0)
    world, pts = scenes.pointcloud_world(np.random.default_rng(1), 3000)
    pts = np.concatenate([pts, np.array([[2e4, 0, 0], [0, 0, np.inf], [np.nan, 0, 0]], np.float32)])
    ctx = build_collision_context(robot, world)
    if checker != "binary":
        # no self pair or world in the gate's way: what is left to compare is the cloud
        ctx.update({k: v[:0] for k, v in ctx.items() if k.startswith("world_")})
        for k in ("self_pairs", "coarse_self_pairs", "self_pair_ranges"):
            ctx[k] = ctx[k][:0]
    bare = {k: v for k, v in ctx.items() if k not in COARSE}
    cloud = PointCloud(pts, r_env, cell)
    rng = np.random.default_rng(2)
    a = PointCloudChecker(ctx, robot.dim, checker)
    b = PointCloudChecker(bare, robot.dim, "binary")
    for n, g in ((1, 1), (31, 1), (33, 2), (700, 3)):
        e = rng.uniform(robot.lower, robot.upper, (n, g, robot.dim)).astype(np.float32)
        e[0, 0, 3] = np.nan
        x = a.check_edges_collision_free(e, None, cloud, r_env).cpu().numpy()
        assert np.array_equal(x, b.check_edges_collision_free(e, None, cloud, r_env).cpu().numpy()), (n, g)
    q = rng.uniform(-1.0, 1.0, (2, 3, robot.dim)).astype(np.float32)
    kw = dict(max_iterations=40, num_new_samples=1, max_nodes=512, min_vals=robot.lower, max_vals=robot.upper,
              tail_explorers=False, point_cloud=cloud)
    for x, y in zip(prrtc_plan_batch(q[0], q[1][:, None], collision_context=ctx, collision_checker=checker, **kw),
                    prrtc_plan_batch(q[0], q[1][:, None], collision_context=bare, **kw)):
        assert (x.solved, x.tree_a_size, x.tree_b_size, x.iterations) == (y.solved, y.tree_a_size, y.tree_b_size,
                                                                          y.iterations)
        assert np.array_equal(x.tree_a_configs.cpu().numpy().view(np.uint32), y.tree_a_configs.cpu().numpy().view(np.uint32))


@pytest.mark.parametrize("mode", [0, 1, 2, 3])
@pytest.mark.parametrize("form", FORMS)
def test_culled_verdicts_equal_full_sweep(cuda, form, mode):
    """The default path against the full sweep, over scenes at the edge of what is culled, counts around a warp's
    share and a configuration that is not a number."""
    from prrtc_b200.collision import CollisionChecker

    robot, ctx = _odd_scene(form, np.random.default_rng(21))
    chk = CollisionChecker(ctx, robot.dim, CHECKERS[mode], 0.02, device=cuda)
    rng = np.random.default_rng(22)
    for n in (1, 5, 127, 3001):
        q = rng.uniform(robot.lower, robot.upper, (n, robot.dim)).astype(np.float32)
        q[n // 2, 2] = (np.nan, np.inf, 1e30, 0.1)[n % 4]
        assert np.array_equal(chk.check(q).cpu().numpy(), chk.check(q, full_sweep=True).cpu().numpy()), n


@pytest.mark.parametrize("mode", [0, 1, 3])
def test_batched_scenes_equal_one_by_one(cuda, mode):
    """One launch over many scenes (uneven shares, an empty one, one that the culled checker does not take) against
    a checker per scene."""
    import ctypes as C

    import torch

    from prrtc_b200 import _lib
    from prrtc_b200.collision import CollisionChecker
    from prrtc_b200.smoothing import _BatchScenes

    robot = scenes.arm(0)
    rng = np.random.default_rng(7)
    ctxs = [build_collision_context(robot, w) for w in (
        scenes.tabletop_world(rng), scenes.spheres_world(rng, 16), {}, scenes.uneven_world(rng),
        {"world_halfspaces": np.array([[0, 0, 3.0, 0, 0, 0.1]], np.float32)}, scenes.tabletop_world(rng))]
    share = [1, 300, 0, 37, 64, 5]
    off = np.concatenate([[0], np.cumsum(share)]).astype(np.int32)
    q = torch.from_numpy(rng.uniform(robot.lower, robot.upper, (off[-1], robot.dim)).astype(np.float32)).to(cuda)
    sc = _BatchScenes(ctxs, cuda)
    v = torch.full((int(off[-1]),), -1, dtype=torch.int32, device=cuda)
    offsets = torch.from_numpy(off).to(cuda)
    lib = _lib.load()
    ws = torch.empty(lib.prrtc_b200_check_configs_batch_workspace_size(C.byref(sc.bi)), dtype=torch.uint8, device=cuda)
    _lib.check(lib.prrtc_b200_check_configs_batch(C.byref(sc.bi), robot.dim, q.data_ptr(), offsets.data_ptr(), int(off[-1]),
                                                  mode, 0.02, v.data_ptr(), ws.data_ptr(), ws.numel(),
                                                  torch.cuda.current_stream().cuda_stream), "check_configs_batch")
    for k, ctx in enumerate(ctxs):
        if share[k]:
            seg = slice(int(off[k]), int(off[k + 1]))
            want = CollisionChecker(ctx, robot.dim, CHECKERS[mode], 0.02, cuda).check(q[seg], full_sweep=True)
            assert torch.equal(v[seg], want), k
