"""The culled checks against the full tests where the pads decide (GPU): primitives of every type and size that graze a
robot sphere, models in metres and in centimetres, boxes that are sheared or stretched, normals of any length,
groups that leave spheres out or hold another frame's.  Verdicts and plans have to be the same bits."""
from __future__ import annotations

import numpy as np
import pytest

from prrtc_b200 import scenes
from prrtc_b200.context import build_collision_context

pytestmark = pytest.mark.gpu

CHECKERS = ["binary", "differentiable", "binary_coarse", "binary_coarse_coop"]
COARSE = ("coarse_sphere_link_idx", "coarse_sphere_local", "coarse_sphere_radius", "fine_link_offsets",
          "coarse_self_pairs", "self_pair_ranges")


def _scaled(ctx: dict, s: float) -> dict:
    """The robot in units of 1/s metres."""
    out = {k: np.array(v) for k, v in ctx.items()}
    out["fk_parent_tf"][:, 4:] *= s
    for k in ("sphere_local", "sphere_radius", "coarse_sphere_local", "coarse_sphere_radius"):
        out[k] = (out[k] * s).astype(np.float32)
    return out


def _frame(rng, u):
    v = np.cross(u, rng.normal(size=3))
    v /= np.linalg.norm(v)
    return v, np.cross(u, v)


def _grazing(form: str, c, r, u, gap, s, rng):
    """A primitive of `form` whose distance from the sphere (c, r) along u is `gap`: its table and its row."""
    v, w = _frame(rng, u)
    if form.startswith("sphere"):
        R = {"sphere_small": 0.03, "sphere_30": 30.0, "sphere_300": 300.0}[form] * s
        return "world_spheres", [*(c + u * (r + R + gap)), R]
    if form.startswith("capsule"):
        R, L = 0.05 * s, (0.4 if form == "capsule" else 500.0) * s
        m = c + u * (r + R + gap) + v * rng.uniform(-0.3, 0.3) * L
        return "world_capsules", [*(m - 0.5 * L * v), *(m + 0.5 * L * v), R]
    if form.startswith("halfspace"):
        n = {"halfspace": 1.0, "halfspace_long": 3.0, "halfspace_short": 0.4}[form] * u
        # n.c - n.p = |n| (c - p).u is compared with r; the point lies anywhere in the plane
        p = c - u * (r + gap) / np.linalg.norm(n) + (v * rng.normal() + w * rng.normal()) * 20 * s
        return "world_halfspaces", [*n, *p]
    h = (500.0 if form == "box_500" else 0.2) * s
    axes = {"box": [u, v, w], "box_500": [u, v, w], "box_sheared": [u + 0.4 * v, v, w - 0.3 * u], "box_long": [2.5 * u, 2.5 * v, 2.5 * w],
            "box_short": [0.3 * u, 0.3 * v, 0.3 * w]}[form]
    a = np.array(axes)
    # along u from the box's centre the first axis coordinate is |a0 . u| t: the face's distance in it is r + gap
    t = (h + r + gap) / float(a[0] @ u)
    return "world_boxes", [*(c + u * t), *a.reshape(-1), h, h * 3, h * 3]


FORMS = ["sphere_small", "sphere_30", "sphere_300", "capsule", "capsule_500", "halfspace", "halfspace_long", "halfspace_short",
         "box", "box_500", "box_sheared", "box_long", "box_short"]


def _scene(orc, form, scale, rng, margin, count=24):
    """A scene of `count` primitives that each graze a sphere of a configuration of their own, and those configurations."""
    robot = scenes.arm(0)
    ctx = _scaled(build_collision_context(robot, {}), scale)
    q = rng.uniform(robot.lower, robot.upper, (count, robot.dim))
    sc = orc.Scene(ctx, robot.dim)
    rows = []
    for x in q:
        F = sc.fk(x).reshape(-1, 12)
        i = int(rng.integers(len(ctx["sphere_radius"])))
        f = F[ctx["sphere_link_idx"][i]]
        c = f[:9].reshape(3, 3) @ ctx["sphere_local"][i].astype(np.float64) + f[9:]
        u = rng.normal(size=3)
        u /= np.linalg.norm(u)
        gap = rng.choice([0.0, 1e-7, -1e-7, 1e-6, -1e-6, 1e-5, -1e-5, 1e-4, -1e-4]) * scale
        key, row = _grazing(form, c, float(ctx["sphere_radius"][i]) + margin, u, gap, scale, rng)
        rows.append(row)
    ctx[key] = np.array(rows, np.float32)
    return robot, ctx, q.astype(np.float32)


@pytest.mark.parametrize("mode", [0, 1, 2, 3])
@pytest.mark.parametrize("scale", [1.0, 100.0])
@pytest.mark.parametrize("form", FORMS)
def test_grazing_primitives(cuda, orc, form, scale, mode):
    """One scene per few primitives (those of many hide one another), each configuration and its neighbours."""
    from prrtc_b200.collision import CollisionChecker

    rng = np.random.default_rng([FORMS.index(form), int(scale), mode])
    margin = 0.02 * scale if mode == 1 else 0.0
    for count in (1, 1, 1, 2, 24):
        robot, ctx, q = _scene(orc, form, scale, rng, margin, count)
        if mode < 2:  # most configurations touch themselves: leave the world alone to decide
            for k in ("self_pairs", "coarse_self_pairs", "self_pair_ranges"):
                ctx[k] = ctx[k][:0]
        near = np.concatenate([q] + [np.repeat(q, 40, 0) + rng.normal(0, e, (40 * len(q), robot.dim))
                                     for e in (1e-6, 1e-4, 1e-2)]).astype(np.float32)
        chk = CollisionChecker(ctx, robot.dim, CHECKERS[mode], margin, device=cuda)
        assert np.array_equal(chk.check(near).cpu().numpy(), chk.check(near, full_sweep=True).cpu().numpy()), count


def _odd(form, rng):
    robot = scenes.arm(0)
    ctx = build_collision_context(robot, scenes.tabletop_world(rng))
    if form == "floor_500":
        ctx["world_boxes"] = np.concatenate([ctx["world_boxes"], np.array(
            [[0, 0, -500.3, 1, 0, 0, 0, 1, 0, 0, 0, 1, 500, 500, 500]], np.float32)])
    elif form == "first_sphere_left_out":
        ctx["fine_link_offsets"] = ctx["fine_link_offsets"] + (np.arange(len(ctx["fine_link_offsets"])) == 0).astype(np.int32)
    elif form == "last_spheres_left_out":
        f = ctx["fine_link_offsets"].copy()
        f[-1] -= 3
        ctx["fine_link_offsets"] = f
    elif form == "all_but_one_link":
        f = ctx["fine_link_offsets"].copy()
        f[:3] = f[3]
        f[4:] = f[4]
        ctx["fine_link_offsets"] = f
    elif form == "another_frame":
        f = ctx["sphere_link_idx"].copy()
        f[10::17] = 0
        ctx["sphere_link_idx"] = f
    elif form == "no_ranges":
        f = ctx["fine_link_offsets"].copy()
        f[2] = f[3] + 2
        ctx["fine_link_offsets"] = f
    elif form == "nan_axis":
        b = ctx["world_boxes"].copy()
        b[0, 3] = np.nan
        b[1, 7] = np.inf
        ctx["world_boxes"] = b
        ctx["world_halfspaces"] = np.array([[0, 0, np.inf, 0, 0, -3], [0, np.nan, 1, 0, 0, -3], [0, 0, 1, 0, 0, -0.05]], np.float32)
    elif form == "negative_radii":
        ctx["sphere_radius"] = ctx["sphere_radius"] * np.where(np.arange(len(ctx["sphere_radius"])) % 5 == 2, -1, 1).astype(np.float32)
        ctx["coarse_sphere_radius"] = ctx["coarse_sphere_radius"] * np.where(np.arange(len(ctx["coarse_sphere_radius"])) == 3, -1, 1).astype(np.float32)
    elif form == "centimetres":
        s = 100.0
        ctx = _scaled(ctx, s)
        for k in ("world_spheres", "world_capsules"):
            ctx[k] = (ctx[k] * s).astype(np.float32)
        ctx["world_boxes"][:, :3] *= s
        ctx["world_boxes"][:, 12:] *= s
        ctx["world_halfspaces"][:, 3:] *= s
    elif form == "stretched":
        ctx["world_boxes"] = ctx["world_boxes"].copy()
        ctx["world_boxes"][::2, 3:12] *= 1.7
        ctx["world_boxes"][1::3, 3:6] += 0.5 * ctx["world_boxes"][1::3, 6:9]
    return robot, ctx


ODD = ["plain", "floor_500", "first_sphere_left_out", "last_spheres_left_out", "all_but_one_link", "another_frame", "no_ranges",
       "nan_axis", "negative_radii", "centimetres", "stretched"]


@pytest.mark.parametrize("mode", [0, 1, 2, 3])
@pytest.mark.parametrize("form", ODD)
def test_verdicts(cuda, form, mode):
    from prrtc_b200.collision import CollisionChecker

    robot, ctx = _odd(form, np.random.default_rng(31))
    chk = CollisionChecker(ctx, robot.dim, CHECKERS[mode], 0.02, device=cuda)
    rng = np.random.default_rng(32)
    for n in (1, 33, 6000):
        q = rng.uniform(robot.lower, robot.upper, (n, robot.dim)).astype(np.float32)
        assert np.array_equal(chk.check(q).cpu().numpy(), chk.check(q, full_sweep=True).cpu().numpy()), n


@pytest.mark.parametrize("problems,threads", [(5, 0), (5, 256), (310, 0), (310, 256), (310, 64)])
@pytest.mark.parametrize("form", ODD)
def test_plans(cuda, form, problems, threads):
    """One explorer per problem, flat checker: the scene with its coarse model (culled edge checks, a CTA of 512 or 256
    threads per explorer, one or two of them per SM) and without it (the general checker)."""
    from prrtc_b200 import prrtc_plan_batch

    robot, ctx = _odd(form, np.random.default_rng(33))
    bare = {k: v for k, v in ctx.items() if k not in COARSE}
    q = np.random.default_rng(34).uniform(-1.2, 1.2, (2, problems, robot.dim)).astype(np.float32)
    kw = dict(max_iterations=25, num_new_samples=1, max_nodes=256, min_vals=robot.lower, max_vals=robot.upper,
              collision_checker="binary", edge_resolution=0.02, tail_explorers=False)
    got = prrtc_plan_batch(q[0], q[1][:, None], collision_context=[ctx] * problems, threads_per_explorer=threads, **kw)
    want = prrtc_plan_batch(q[0], q[1][:, None], collision_context=[bare] * problems, threads_per_explorer=128, **kw)
    for a, b in zip(got, want):
        assert (a.solved, a.tree_a_size, a.tree_b_size, a.iterations) == (b.solved, b.tree_a_size, b.tree_b_size, b.iterations)
        for x, y in ((a.tree_a_configs, b.tree_a_configs), (a.tree_b_configs, b.tree_b_configs)):
            assert np.array_equal(x.cpu().numpy().view(np.uint32), y.cpu().numpy().view(np.uint32))
