"""Performance cases: what a user's program has this planner do, through its public entry points.

Robots and worlds are the ones of the benchmark workloads (``prrtc_b200.scenes``): the 7-joint arm with
56 spheres and 960 self pairs, and the dual arm with 14 actuated and 4 mimic joints and 120 spheres.
Configurations, start / goal pairs and paths are drawn from the case's seed and kept when a plain torch
check (below, independent of the kernels) finds them free.

Planning comes in two forms.  By default the explorers of a problem race, so the path, its cost and the
tree sizes are those of whichever explorer came first and differ from run to run; a case of that form
returns what does not depend on the race, the solved flags and the ends of the paths that the problem
itself fixes.  With one explorer per problem and no tail explorers a plan is reproducible, and such a case
returns everything: flags, paths, costs, tree sizes and iteration counts.
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import prrtc_b200 as P
from prrtc_b200 import collision, scenes, smoothing
from prrtc_b200.context import build_collision_context, with_world


def listed():
    return [
        # One motion query of an interactive program: 16 spheres, defaults otherwise (128 explorers, binary
        # checker, 16 waypoints per edge).  Latency is what counts.
        dict(name="plan_single", kind="plan", robot="arm", world="spheres16", batch=0, explorers=128, checker="binary",
             resolution=0.0, threads=0, chunk=0, max_nodes=65536, iterations=10000),
        # The benchmark's headline call: 512 problems of uneven worlds and tree capacities in one batch,
        # host inputs, paths read back, the settings its tuner picks.
        dict(name="plan_batch_uneven", kind="plan", robot="arm", world="uneven", batch=512, explorers=2,
             checker="binary_coarse_coop", resolution=0.01, threads=256, chunk=64, max_nodes=0, iterations=10000),
        # Reproducible plans (one explorer each) of a tabletop batch with 4 goals per problem.
        dict(name="plan_batch_tabletop", kind="plan", robot="arm", world="tabletop", batch=200, explorers=1,
             checker="binary_coarse_coop", resolution=0.01, threads=256, chunk=64, max_nodes=16384, iterations=2000),
        # Reproducible dual-arm plans in the large world.
        dict(name="plan_batch_dual_arm", kind="plan", robot="dual_arm", world="large", batch=61, explorers=1,
             checker="binary_coarse_coop", resolution=0.01, threads=256, chunk=16, max_nodes=16384, iterations=300),
        # Rejection sampling of free configurations, 256 candidates a call (what the problem generators do).
        dict(name="check_256", kind="check", robot="arm", world="tabletop", n=256, checker="binary"),
        # Bulk labelling of configurations, the checker benchmark's size.
        dict(name="check_1m", kind="check", robot="arm", world="tabletop", n=1 << 20, checker="binary"),
        # The coarse-gated checker on the dual arm, an odd count.
        dict(name="check_dual_arm", kind="check", robot="dual_arm", world="large", n=50021, checker="binary_coarse_coop"),
        # One batch of edges of the host-driven planner: 128 samples x 16 waypoints against a scanned cloud.
        dict(name="edges_cloud", kind="edges", n=128, granularity=16, points=20000, fresh_cloud=False),
        # Nearest neighbour of a batch of samples in a large tree (117 MB).
        dict(name="nearest_4m", kind="nearest", dim=7, capacity=1 << 22, size=(1 << 22) - 4321, batch=64),
        # Link frames of a batch of dual-arm configurations.
        dict(name="fk_dual_arm", kind="fk", robot="dual_arm", n=65537),
        # One optimisation step on a batch of planned paths: cost and gradient through autograd.
        dict(name="smooth_cost", kind="smooth", robot="arm", world="tabletop", paths=512, waypoints=64),
        # Post-processing of a small batch of plans, each in its own world: the whole smoothing call.
        dict(name="smooth_paths", kind="smooth_paths", robot="arm", world="tabletop", paths=32, waypoints=64, steps=50),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["plan", "plan", "check", "check", "edges", "nearest", "fk", "smooth", "smooth_paths"])
    checker = rng.choice(["binary", "differentiable", "binary_coarse", "binary_coarse_coop"])
    if kind == "plan":
        world = rng.choice(["spheres16", "uneven", "tabletop"])
        return dict(kind="plan", robot="arm", world=world, batch=_log_int(rng, 1, 150), explorers=1, checker=checker,
                    resolution=rng.choice([0.0, 0.01, 0.02]), threads=rng.choice([0, 64, 256]),
                    chunk=rng.choice([0, 32, 64]), max_nodes=rng.choice([4096, 16384, 20001]), iterations=500)
    if kind == "check":
        robot = rng.choice(["arm", "arm", "dual_arm"])
        world = "large" if robot == "dual_arm" else rng.choice(["spheres16", "uneven", "tabletop"])
        return dict(kind="check", robot=robot, world=world, checker=checker,
                    n=_log_int(rng, 33, 60000 if robot == "dual_arm" else 1000000))
    if kind == "edges":
        return dict(kind="edges", n=_log_int(rng, 33, 8000), granularity=rng.choice([1, 8, 16, 33]),
                    points=_log_int(rng, 1000, 100000), fresh_cloud=rng.random() < 0.5)
    if kind == "nearest":
        capacity = _log_int(rng, 1000, 1 << 22)
        return dict(kind="nearest", dim=rng.choice([6, 7, 14]), capacity=capacity,
                    size=max(1, int(capacity * rng.uniform(0.3, 1.0))), batch=_log_int(rng, 1, 64))
    if kind == "fk":
        return dict(kind="fk", robot=rng.choice(["arm", "dual_arm"]), n=_log_int(rng, 1, 65000))
    if kind == "smooth":
        robot = rng.choice(["arm", "arm", "dual_arm"])
        waypoints = rng.choice([32, 64, 96, 101])
        most = (4000 if robot == "dual_arm" else 32000) // waypoints
        return dict(kind="smooth", robot=robot, world="large" if robot == "dual_arm" else "tabletop",
                    paths=_log_int(rng, 1, most), waypoints=waypoints)
    return dict(kind="smooth_paths", robot="arm", world=rng.choice(["spheres16", "tabletop"]), paths=_log_int(rng, 1, 24),
                waypoints=rng.choice([32, 48, 64]), steps=rng.choice([20, 50]))


# ----------------------------------------------------------------------------- robots, worlds, plain torch geometry

_WORLDS = {"spheres16": lambda rng: scenes.spheres_world(rng, 16), "uneven": scenes.uneven_world,
           "tabletop": scenes.tabletop_world, "large": scenes.large_world}
_KEYS = ("world_spheres", "world_capsules", "world_boxes", "world_halfspaces")


@functools.lru_cache(maxsize=None)
def _robot(name):
    robot = scenes.dual_arm(0) if name == "dual_arm" else scenes.arm(0)
    return robot, build_collision_context(robot)


def _dev():
    return torch.device("cuda")


class _Model:
    """Robot tables as torch tensors; FK, sphere centres and clearances by plain torch."""

    def __init__(self, robot_name, dtype):
        robot, ctx = _robot(robot_name)
        dev = _dev()

        def t(x, dt=dtype):
            return torch.as_tensor(np.asarray(x), device=dev).to(dt)

        self.dim, self.J, self.dtype = robot.dim, robot.n_joints, dtype
        self.parent = [int(p) for p in ctx["fk_parent_idx"]]
        self.act = [int(a) for a in ctx["fk_act_idx"]]
        self.mimic = [(int(m), float(k), float(o)) for m, k, o in
                      zip(ctx["fk_mimic_act_idx"], ctx["fk_mimic_mul"], ctx["fk_mimic_off"])]
        assert not np.any(ctx["fk_twists"][:, :3]), "these robots have revolute joints only"
        axis = t(ctx["fk_twists"][:, 3:])
        z = torch.zeros_like(axis[:, 0])
        self.K = torch.stack([z, -axis[:, 2], axis[:, 1], axis[:, 2], z, -axis[:, 0], -axis[:, 1], axis[:, 0], z],
                             1).reshape(-1, 3, 3)
        q = t(ctx["fk_parent_tf"][:, :4], torch.float64)
        q = q / q.norm(dim=1, keepdim=True)
        w, x, y, zz = q.unbind(1)
        self.PR = torch.stack([1 - 2 * (y * y + zz * zz), 2 * (x * y - w * zz), 2 * (x * zz + w * y),
                               2 * (x * y + w * zz), 1 - 2 * (x * x + zz * zz), 2 * (y * zz - w * x),
                               2 * (x * zz - w * y), 2 * (y * zz + w * x), 1 - 2 * (x * x + y * y)],
                              1).reshape(-1, 3, 3).to(dtype)
        self.Pt = t(ctx["fk_parent_tf"][:, 4:])
        self.frame = t(ctx["sphere_link_idx"], torch.int64)
        self.local, self.radius = t(ctx["sphere_local"]), t(ctx["sphere_radius"])
        self.pairs = t(ctx["self_pairs"], torch.int64)
        self.S, self.Q = self.radius.numel(), self.pairs.shape[0]
        self.links, self.link_pairs = len(ctx["coarse_sphere_radius"]), len(ctx["coarse_self_pairs"])

    def fk(self, q):
        """Rotations [n, J, 3, 3] and origins [n, J, 3] of configurations [n, dim]."""
        q = q.to(self.dtype)
        eye = torch.eye(3, dtype=self.dtype, device=q.device)
        R, T = [], []
        for j in range(self.J):
            m, mul, off = self.mimic[j]
            v = mul * q[:, m] + off if m >= 0 else (q[:, self.act[j]] if self.act[j] >= 0 else torch.zeros_like(q[:, 0]))
            K = self.K[j]
            E = eye + v.sin()[:, None, None] * K + (1 - v.cos())[:, None, None] * (K @ K)
            r, t = self.PR[j] @ E, self.Pt[j].expand(q.shape[0], 3)
            p = self.parent[j]
            if p >= 0:
                r, t = R[p] @ r, (R[p] @ t[:, :, None])[:, :, 0] + T[p]
            R.append(r)
            T.append(t)
        return torch.stack(R, 1), torch.stack(T, 1)

    def centres(self, q):
        R, T = self.fk(q)
        return (R[:, self.frame] @ self.local[:, :, None])[..., 0] + T[:, self.frame]

    def world_distances(self, c, w):
        """Signed distances of sphere centres c [B, n, 3] (n spheres of the robot, repeated) to every
        primitive of the padded worlds w, per primitive type: list of [B, n, count]."""
        r = self.radius.repeat(c.shape[1] // self.S)[None, :, None]
        out = []
        ws, wc, wb, wh = (w[k] for k in _KEYS)
        if ws.shape[1]:
            out.append(_norm(c[:, :, None] - ws[:, None, :, :3]) - ws[:, None, :, 3] - r)
        if wc.shape[1]:
            p, d = wc[:, None, :, :3], (wc[..., 3:6] - wc[..., :3])[:, None]
            e = c[:, :, None] - p
            t = ((e * d).sum(-1) / (d * d).sum(-1).clamp_min(1e-30)).clamp(0, 1)
            out.append(_norm(e - t[..., None] * d) - wc[:, None, :, 6] - r)
        if wb.shape[1]:
            e = c[:, :, None] - wb[:, None, :, :3]
            a = wb[..., 3:12].reshape(wb.shape[0], 1, wb.shape[1], 3, 3)
            l = (a * e[..., None, :]).sum(-1)
            q = l.abs() - wb[:, None, :, 12:15]
            outside = _norm(q.clamp_min(0))
            out.append(torch.where(q.amax(-1) > 0, outside, q.amax(-1)) - r)
        if wh.shape[1]:
            out.append((wh[:, None, :, :3] * (c[:, :, None] - wh[:, None, :, 3:6])).sum(-1) - r)
        return out

    def self_distances(self, c):
        """Signed distances [..., pairs] of the self pairs from centres [..., S, 3]."""
        i, j = self.pairs[:, 0], self.pairs[:, 1]
        return _norm(c[..., i, :] - c[..., j, :]) - self.radius[i] - self.radius[j]

    def free(self, q, w, clearance=1e-3):
        """Whether configurations [B, C, dim] are free of the padded worlds w (of B, or of 1 for all)."""
        B, C, _ = q.shape
        n = max(1, sum(w[k].shape[1] for k in _KEYS))
        step = max(1, int(6e7 // (B * self.S * n)))
        ok = []
        for a in range(0, C, step):
            x = q[:, a:a + step]
            c = self.centres(x.reshape(-1, self.dim))
            f = (self.self_distances(c) > clearance).all(-1).reshape(B, -1) if self.Q else True
            for d in self.world_distances(c.reshape(B, -1, 3), w):
                f = f & (d > clearance).all(-1).reshape(B, x.shape[1], self.S).all(-1)
            ok.append(f)
        return torch.cat(ok, 1)


def _norm(v):
    s = (v * v).sum(-1)
    return torch.where(s > 0, s.clamp_min(1e-60 if v.dtype == torch.float64 else 1e-30).sqrt(), s)


def _padded(worlds, dtype):
    """The worlds as padded tensors [B, most, features]; padding rows are far-away primitives of size 0."""
    out = {}
    for k, width in zip(_KEYS, (4, 7, 15, 6)):
        far = np.zeros(width)
        far[:3] = (0, 0, 1) if k == "world_halfspaces" else 1e3
        far[3:6] = (0, 0, -1e3) if k == "world_halfspaces" else (1e3 if k == "world_capsules" else 0.0)
        if k == "world_spheres":
            far[3] = 0.0
        if k == "world_boxes":
            far[3:12] = np.eye(3).reshape(-1)
        a = np.tile(far, (len(worlds), max(len(w[k]) for w in worlds), 1))
        for i, w in enumerate(worlds):
            a[i, :len(w[k])] = w[k]
        out[k] = torch.as_tensor(a, device=_dev()).to(dtype)
    return out


def _uniform(gen, shape, lo=0.0, hi=1.0):
    return lo + (hi - lo) * torch.rand(shape, generator=gen, device=_dev())


def _generator(seed):
    return torch.Generator(device=_dev()).manual_seed(int(seed))


def _free_configs(model, worlds, count, gen):
    """[B, count, dim] free configurations, uniform within the joint limits."""
    B = len(worlds)
    w = _padded(worlds, model.dtype)
    got = torch.zeros((B, count, model.dim), device=_dev())
    have = torch.zeros(B, dtype=torch.int64, device=_dev())
    for _ in range(40):
        rows = torch.nonzero(have < count)[:, 0]
        if not rows.numel():
            return got
        tries = max(64, 2 * count)
        q = _uniform(gen, (rows.numel(), tries, model.dim), -scenes.ARM_LIMIT, scenes.ARM_LIMIT)
        ok = model.free(q, {k: v[rows] for k, v in w.items()})
        slot = have[rows, None] + ok.cumsum(1) - 1
        take = ok & (slot < count)
        r, c = torch.nonzero(take, as_tuple=True)
        got[rows[r], slot[r, c]] = q[r, c]
        have[rows] = torch.clamp(have[rows] + ok.sum(1), max=count)
    raise RuntimeError("could not sample free configurations")


def _free_paths(model, worlds, count, gen):
    """`count` collision-free polylines [L_i, dim] with steps of at most 0.5 rad, as the planner returns
    them: path i in worlds[i] (or in the only world).  Persistent random walks of 6 to 20 vertices."""
    w = _padded(worlds, model.dtype)
    shared = len(worlds) == 1
    start = _free_configs(model, worlds, count if shared else 1, gen)
    at = (start[0] if shared else start[:, 0]).clone()
    lengths = torch.randint(6, 21, (count,), generator=gen, device=_dev()).tolist()
    way = torch.randn((count, model.dim), generator=gen, device=_dev())
    nodes, tries, ts = [at], 8, torch.linspace(0.2, 1.0, 5, device=_dev())
    for _ in range(19):
        d = way[:, None] / way.norm(dim=-1)[:, None, None] + 0.5 * torch.randn((count, tries, model.dim), generator=gen,
                                                                              device=_dev())
        d = 0.5 * d / d.norm(dim=-1, keepdim=True)
        end = at[:, None] + d
        inside = (end.abs() <= scenes.ARM_LIMIT).all(-1)
        q = at[:, None, None] + ts[None, None, :, None] * d[:, :, None]
        q = q.reshape(1, -1, model.dim) if shared else q.reshape(count, -1, model.dim)
        ok = model.free(q, w).reshape(count, tries, -1).all(-1) & inside
        pick = ok.to(torch.int8).argmax(1)
        moved = ok.any(1)
        step = d[torch.arange(count, device=_dev()), pick] * moved[:, None]
        at = at + step
        way = torch.where(moved[:, None], step, torch.randn((count, model.dim), generator=gen, device=_dev()))
        nodes.append(at)
    nodes = torch.stack(nodes, 1).cpu().numpy()
    out = []
    for p, n in zip(nodes, lengths):
        p = p[:n]
        keep = np.concatenate([[True], np.abs(np.diff(p, axis=0)).max(1) > 0])
        p = p[keep]
        out.append(p if len(p) > 1 else np.repeat(p, 2, 0))
    return out


def _worlds(name, count, seed):
    return [_WORLDS[name](np.random.default_rng([seed, i])) for i in range(count)]


# ----------------------------------------------------------------------------- the cases

def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return state["run"](state)


def work(case):
    return _WORK[case["kind"]](case)


def exact(case, seed):
    f = _EXACT.get(case["kind"])
    return f(case, seed) if f else None


def _mean_world(name):
    """Mean primitive counts (spheres, capsules, boxes, halfspaces) of a world."""
    return {"spheres16": (16, 0, 0, 0), "uneven": (66, 0, 16, 0), "tabletop": (32, 8, 20, 1), "large": (256, 0, 64, 1)}[name]


def _config_flops(robot_name, world):
    """Operations that one verdict cannot do without: link frames, sphere centres, and every link's bounding
    sphere against every primitive and every link pair's (finer tests only where those touch)."""
    robot, ctx = _robot(robot_name)
    ns, nc, nb, nh = _mean_world(world)
    links, pairs = len(ctx["coarse_sphere_radius"]), len(ctx["coarse_self_pairs"])
    return (robot.n_joints * 153 + len(ctx["sphere_radius"]) * 18 + links * (8 * ns + 23 * nc + 26 * nb + 6 * nh) +
            pairs * 11)


# -- planning

_LONGEST = 512  # waypoints; paths of a few dozen are usual


def _prepare_plan(case, seed):
    model = _Model(case["robot"], torch.float32)
    robot, base = _robot(case["robot"])
    B = max(1, case["batch"])
    worlds = _worlds(case["world"], B, seed)
    rng = np.random.default_rng([seed, 1 << 20])
    most = {"spheres16": 1, "tabletop": 4, "uneven": 8, "large": 4}[case["world"]]
    goals_of = rng.integers(1, most + 1, size=B) if case["world"] in ("uneven", "large") else np.full(B, most)
    q = _free_configs(model, worlds, 1 + most, _generator(seed)).cpu().numpy()
    nodes = case["max_nodes"]
    if nodes == 0:  # a tree capacity per problem, by the size of its world
        nodes = []
        for w in worlds:
            n = len(w["world_spheres"]) + len(w["world_boxes"])
            nodes.append(scenes.BUCKETS[0 if n < 48 else (1 if n < 112 else 2)])
    contexts = [with_world(base, w) for w in worlds]
    kw = dict(max_iterations=case["iterations"], num_new_samples=case["explorers"], max_nodes=nodes,
              min_vals=robot.lower, max_vals=robot.upper, collision_checker=case["checker"],
              edge_resolution=case["resolution"], threads_per_explorer=case["threads"], waypoint_chunk=case["chunk"])
    if case["batch"] == 0:
        return dict(run=_run_plan_single, start=q[0, 0], goals=q[0, 1:], context=contexts[0], kw=kw)
    kw.update(goal_counts=goals_of.tolist(), tail_explorers=case["explorers"] > 1, return_trees=False, paths_on_host=True)
    return dict(run=_run_plan_batch if case["explorers"] > 1 else _run_plan_reproducible, start=q[:, 0], goals=q[:, 1:],
                context=contexts, kw=kw)


def _run_plan_single(s):
    r = P.prrtc_plan(s["start"], s["goals"], collision_context=s["context"], **s["kw"])
    return {"solved": r.solved, "ends": torch.stack([r.path[0], r.path[-1]]) if r.solved else torch.zeros(2, len(s["start"]))}


def _run_plan_batch(s):
    results = P.prrtc_plan_batch(s["start"], s["goals"], collision_context=s["context"], **s["kw"])
    return {"solved": np.array([r.solved for r in results]),
            "starts": np.stack([r.path[0].numpy() if r.solved else 0 * s["start"][0] for r in results])}


def _run_plan_reproducible(s):
    results = P.prrtc_plan_batch(s["start"], s["goals"], collision_context=s["context"], **s["kw"])
    paths = np.zeros((len(results), _LONGEST, s["start"].shape[1]), np.float32)
    for k, r in enumerate(results):
        if r.solved:
            paths[k, :len(r.path)] = r.path.numpy()
    return {"solved": np.array([r.solved for r in results]),
            "sizes": np.array([(r.tree_a_size, r.tree_b_size, r.iterations) for r in results]),
            "lengths": np.array([len(r.path) if r.solved else 0 for r in results]),
            "costs": np.array([r.cost for r in results], np.float32),
            "paths": paths}


def _work_plan(case):
    # inputs and paths, and the waypoints of one straight motion (5 rad, every 0.01 rad) per problem
    B = max(1, case["batch"])
    ns, nc, nb, nh = _mean_world(case["world"])
    world = 4 * (4 * ns + 7 * nc + 15 * nb + 6 * nh)
    return {"bytes": B * (world + 4 * 16 * 30), "flops": B * 500.0 * _config_flops(case["robot"], case["world"])}


# -- collision checking

def _prepare_check(case, seed):
    robot, base = _robot(case["robot"])
    context = with_world(base, _worlds(case["world"], 1, seed)[0])
    checker = collision.CollisionChecker(context, robot.dim, case["checker"])
    q = _uniform(_generator(seed), (case["n"], robot.dim), -scenes.ARM_LIMIT, scenes.ARM_LIMIT)
    return dict(run=lambda s: s["checker"].check(s["q"]), checker=checker, q=q)


def _work_check(case):
    dim = _robot(case["robot"])[0].dim
    return {"bytes": case["n"] * 4 * (dim + 1), "flops": case["n"] * float(_config_flops(case["robot"], case["world"]))}


def _prepare_edges(case, seed):
    robot, base = _robot("arm")
    world, points = scenes.pointcloud_world(np.random.default_rng([seed, 0]), case["points"])
    context = with_world(base, world)
    checker = P.PointCloudChecker(context, robot.dim)
    gen = _generator(seed)
    a = _uniform(gen, (case["n"], 1, robot.dim), -scenes.ARM_LIMIT, scenes.ARM_LIMIT)
    d = torch.randn((case["n"], 1, robot.dim), generator=gen, device=_dev())
    t = torch.linspace(0.0, 1.0, case["granularity"], device=_dev())[None, :, None]
    edges = a + 0.5 * t * d / d.norm(dim=-1, keepdim=True)
    points = torch.as_tensor(points, device=_dev())
    cloud = None if case["fresh_cloud"] else P.PointCloud(points, r_env=0.01)
    return dict(run=_run_edges, checker=checker, edges=edges.contiguous(), points=points, cloud=cloud)


def _run_edges(s):
    # a program that gets a new scan for every batch of edges hashes it first
    cloud = s["cloud"] if s["cloud"] is not None else P.PointCloud(s["points"], r_env=0.01)
    return s["checker"].check_edges_collision_free(s["edges"], None, cloud, 0.01)


def _work_edges(case):
    n = case["n"] * case["granularity"]
    # the analytic part of the tabletop scene, and a sphere's share of the cloud (a 27-cell neighbourhood)
    return {"bytes": n * 4 * 7 + case["points"] * 16, "flops": float(n) * (_config_flops("arm", "tabletop") + 56 * 30)}


# -- nearest neighbour

def _nearest_inputs(case, seed):
    gen = _generator(seed)
    tree = _uniform(gen, (case["dim"], case["capacity"]), -scenes.ARM_LIMIT, scenes.ARM_LIMIT)
    return tree, _uniform(gen, (case["batch"], case["dim"]), -scenes.ARM_LIMIT, scenes.ARM_LIMIT)


def _prepare_nearest(case, seed):
    tree, q = _nearest_inputs(case, seed)
    return dict(run=lambda s: P.prrtc_nearest_neighbor(s["tree"], s["q"], s["size"]), tree=tree, q=q, size=case["size"])


def _work_nearest(case):
    return {"bytes": 4 * case["dim"] * case["size"], "flops": 3.0 * case["dim"] * case["size"] * case["batch"]}


def _exact_nearest(case, seed):
    tree, q = _nearest_inputs(case, seed)
    t = tree[:, :case["size"]].double().T.contiguous()
    dist, idx = zip(*((lambda d: (d.min(), d.argmin()))((t - x).square().sum(1).sqrt()) for x in q.double()))
    return torch.stack(dist), torch.stack(idx)


# -- forward kinematics

def _fk_inputs(case, seed):
    robot, context = _robot(case["robot"])
    return context, _uniform(_generator(seed), (case["n"], robot.dim), -scenes.ARM_LIMIT, scenes.ARM_LIMIT)


def _prepare_fk(case, seed):
    context, q = _fk_inputs(case, seed)
    return dict(run=lambda s: collision.forward_kinematics(s["q"], s["context"]), context=context, q=q)


def _work_fk(case):
    robot, _ = _robot(case["robot"])
    return {"bytes": 4.0 * case["n"] * (robot.dim + 12 * robot.n_joints), "flops": 153.0 * case["n"] * robot.n_joints}


def _exact_fk(case, seed):
    _, q = _fk_inputs(case, seed)
    R, T = _Model(case["robot"], torch.float64).fk(q)  # frame k is joint k for these robots
    return torch.cat([R.reshape(R.shape[0], -1, 9), T], 2)


# -- smoothing

def _smooth_inputs(case, seed):
    model = _Model(case["robot"], torch.float32)
    worlds = _worlds(case["world"], 1, seed)
    paths = _free_paths(model, worlds, case["paths"], _generator(seed))
    x = np.stack([smoothing.resample_path(p, case["waypoints"]) for p in paths])
    return worlds, torch.as_tensor(x, device=_dev())


def _prepare_smooth(case, seed):
    robot, base = _robot(case["robot"])
    worlds, x = _smooth_inputs(case, seed)
    sctx = smoothing.SmoothContext(with_world(base, worlds[0]), robot.dim)
    return dict(run=_run_smooth, sctx=sctx, x=x)


def _run_smooth(s):
    x = s["x"].detach().requires_grad_(True)
    cost = smoothing.smooth_cost(x, s["sctx"])
    cost.sum().backward()
    return {"cost": cost.detach(), "grad": x.grad}


def _work_smooth(case):
    robot, ctx = _robot(case["robot"])
    ns, nc, nb, nh = _mean_world(case["world"])
    n = case["paths"] * case["waypoints"]
    S, Q = len(ctx["sphere_radius"]), len(ctx["self_pairs"])
    # per pair: the distance, one softplus with its derivative (10), and the gradient's accumulation (6)
    pairs = S * (ns * (8 + 16) + nc * (23 + 16) + nb * (26 + 16) + nh * (6 + 16)) + Q * (8 + 22)
    return {"bytes": 4.0 * n * 2 * robot.dim, "flops": float(n) * (pairs + robot.n_joints * 306 + S * 36)}


def _exact_smooth(case, seed):
    worlds, x = _smooth_inputs(case, seed)
    model = _Model(case["robot"], torch.float64)
    w = _padded(worlds, torch.float64)
    pairs = model.S * sum(v.shape[1] for v in w.values()) + model.Q
    if pairs * x.shape[0] * x.shape[1] > 4e8:
        return None
    beta, margin, w_len = 50.0, 0.02, 1.0  # SmoothContext's defaults
    cost, grad = [], []
    step = max(1, int(3e6 // (pairs * x.shape[1])))
    for a in range(0, x.shape[0], step):
        q = x[a:a + step].double().requires_grad_(True)
        c = model.centres(q.reshape(-1, model.dim))
        n = c.shape[0]
        terms = [torch.nn.functional.softplus(beta * (margin - d), threshold=1e9).reshape(n, -1).sum(1) / beta
                 for d in model.world_distances(c.reshape(1, -1, 3), w) + [model.self_distances(c)]]
        total = sum(terms).reshape(q.shape[:2]).sum(1) + w_len * (q[:, 1:] - q[:, :-1]).square().sum((1, 2))
        total.sum().backward()
        cost.append(total.detach())
        grad.append(q.grad)
    return {"cost": torch.cat(cost), "grad": torch.cat(grad)}


def _prepare_smooth_paths(case, seed):
    robot, base = _robot(case["robot"])
    worlds = _worlds(case["world"], case["paths"], seed)
    paths = _free_paths(_Model(case["robot"], torch.float32), worlds, case["paths"], _generator(seed))
    return dict(run=_run_smooth_paths, paths=paths, contexts=[with_world(base, w) for w in worlds],
                lower=robot.lower, upper=robot.upper, kw=dict(waypoints=case["waypoints"], steps=case["steps"]))


def _run_smooth_paths(s):
    out, accepted, before, after = smoothing.smooth_paths_batch(s["paths"], s["contexts"], s["lower"], s["upper"], **s["kw"])
    return {"paths": out, "accepted": accepted, "before": before, "after": after}


def _work_smooth_paths(case):
    one = _work_smooth(case)
    n = case["paths"] * case["waypoints"]
    # the steps, and the re-validation of about 5 rad of each path at 0.01 rad
    return {"bytes": one["bytes"] * case["steps"],
            "flops": one["flops"] * case["steps"] + case["paths"] * 500.0 * _config_flops(case["robot"], case["world"])
            + 10.0 * n * case["steps"]}


_PREPARE = {"plan": _prepare_plan, "check": _prepare_check, "edges": _prepare_edges, "nearest": _prepare_nearest,
            "fk": _prepare_fk, "smooth": _prepare_smooth, "smooth_paths": _prepare_smooth_paths}
_WORK = {"plan": _work_plan, "check": _work_check, "edges": _work_edges, "nearest": _work_nearest, "fk": _work_fk,
         "smooth": _work_smooth, "smooth_paths": _work_smooth_paths}
_EXACT = {"nearest": _exact_nearest, "fk": _exact_fk, "smooth": _exact_smooth}
