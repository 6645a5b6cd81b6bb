"""Post-plan path smoothing with the hand-written adjoint kernel.

``SmoothCost`` is a ``torch.autograd.Function`` whose forward and backward both
come from ``prrtc_b200_smooth_cost_grad`` (one launch computes the cost and the
gradient through FK, recomputing link transforms instead of storing them) -- the
torch counterpart of a ``jax.custom_vjp`` (jax is not installed here).

Cost of a path with W waypoints q_w:
    sum_w sum_pairs softplus_beta(margin - d_pair(q_w)) + w_len * sum_w |q_{w+1} - q_w|^2
over every robot-sphere / world-primitive pair and every self pair.

``smooth_paths`` runs projected gradient steps (endpoints fixed, joint limits
enforced), then re-validates every smoothed path with the exact collision
checker at a fixed joint-space resolution; a path that fails reverts to the
input path (prrtc_plan's RRT-Connect result).
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import torch
from torch.autograd import forward_ad

from . import _lib
from .collision import CollisionChecker
from .device import ROBOT_SPEC, DeviceContext, Stager, as_tensor, cuda_device, ptr, stream_handle, workspace


class SmoothContext:
    """Robot + world tables resident on the device for the smoothing kernel."""

    def __init__(self, collision_context: dict, dim: int, margin: float = 0.02, beta: float = 50.0,
                 w_len: float = 1.0, device=None):
        self.lib = _lib.load()
        self.device = cuda_device(device)
        self.ctx = DeviceContext(collision_context, self.device)
        self.dim = int(dim)
        self.margin, self.beta, self.w_len = float(margin), float(beta), float(w_len)
        self.robot, self.world = self.ctx.robot(), self.ctx.world()
        self.ws = workspace(self.lib.prrtc_b200_smooth_workspace_size(C.byref(self.robot), C.byref(self.world)),
                            self.device)

    def cost_grad(self, waypoints: torch.Tensor, need_grad: bool = True, ordered: bool = False):
        """cost [P] and gradient [P, W, dim], the gradient the same bits in every run
        of the same call; ``ordered``: also whatever paths are beside it, as
        BatchSmoothContext's (descents)."""
        wp = waypoints.detach().to(self.device, torch.float32).contiguous()
        P, W, dim = wp.shape
        cost = torch.empty((P,), dtype=torch.float32, device=self.device)
        grad = torch.empty_like(wp) if need_grad else None
        call = self.lib.prrtc_b200_smooth_cost_grad_ordered if ordered else self.lib.prrtc_b200_smooth_cost_grad
        _lib.check(call(C.byref(self.robot), C.byref(self.world), dim, ptr(wp), P, W, self.margin, self.beta,
                        self.w_len, ptr(cost), ptr(grad), self.ws.data_ptr(), self.ws.numel(), stream_handle()),
                   "prrtc_b200_smooth_cost_grad")
        return cost, grad


class SmoothCost(torch.autograd.Function):
    """cost[P] = smooth collision + length cost of waypoints [P, W, dim]."""

    @staticmethod
    def forward(ctx, waypoints, sctx: SmoothContext):
        cost, grad = sctx.cost_grad(waypoints, need_grad=waypoints.requires_grad)
        ctx.save_for_backward(grad if grad is not None else torch.empty(0))
        return cost

    @staticmethod
    def backward(ctx, gcost):
        (grad,) = ctx.saved_tensors
        return grad * gcost[:, None, None], None


def smooth_cost(waypoints: torch.Tensor, sctx: SmoothContext) -> torch.Tensor:
    return SmoothCost.apply(waypoints, sctx)


def resample_path(path: np.ndarray, W: int) -> np.ndarray:
    """W waypoints along a piecewise-linear path of L vertices.  With L <= W every
    vertex is kept and the W - L extra points are spread over the segments in
    proportion to their lengths (largest remainders first), so the resampled
    polyline is the input path itself -- a smoothing pass that reverts returns
    exactly the planner's path.  With L > W: W points evenly spaced in arc
    length."""
    path = np.asarray(path, dtype=np.float64)
    if path.shape[0] == 1:
        return np.repeat(path, W, 0).astype(np.float32)
    L = path.shape[0]
    if L <= W:
        seg = np.linalg.norm(np.diff(path, axis=0), axis=1)
        extra = W - L
        share = seg / seg.sum() * extra if seg.sum() > 0 else np.full(L - 1, extra / (L - 1))
        n = np.floor(share).astype(np.int64)
        rest = extra - int(n.sum())
        if rest > 0:
            n[np.argsort(-(share - n), kind="stable")[:rest]] += 1
        out = [path[i] + (np.arange(n[i] + 1) / (n[i] + 1))[:, None] * (path[i + 1] - path[i]) for i in range(L - 1)]
        out.append(path[-1:])
        return np.concatenate(out, 0).astype(np.float32)
    seg = np.linalg.norm(np.diff(path, axis=0), axis=1)
    s = np.concatenate([[0.0], np.cumsum(seg)])
    if s[-1] <= 0:
        return np.repeat(path[:1], W, 0).astype(np.float32)
    t = np.linspace(0.0, s[-1], W)
    idx = np.clip(np.searchsorted(s, t, side="right") - 1, 0, path.shape[0] - 2)
    u = ((t - s[idx]) / np.maximum(seg[idx], 1e-12))[:, None]
    out = path[idx] * (1 - u) + path[idx + 1] * u
    out[0], out[-1] = path[0], path[-1]
    return out.astype(np.float32)


def _spread(paths: list, W: int) -> np.ndarray:
    """resample_path of finite float64 paths of 2..W vertices, all at once:
    [P, W, dim], the same bits (32 paths to 64 points: 2.3 -> 0.3 ms against a
    path and a segment at a time)."""
    P, L = len(paths), np.fromiter((p.shape[0] for p in paths), np.int64, len(paths))
    v = np.concatenate(paths, 0)
    first = np.cumsum(L) - L                                     # row of each path's first vertex
    path_of = np.repeat(np.arange(P), L - 1)                     # of each segment
    a = np.arange(path_of.size) + path_of                        # its first vertex's row
    d = v[a + 1] - v[a]
    seg = np.linalg.norm(d, axis=1)
    total = np.array([seg[f:f + n].sum() for f, n in zip(first - np.arange(P), L - 1)])
    extra = (W - L)[path_of]
    with np.errstate(invalid="ignore"):  # 0 / 0 of a path without length
        share = np.where(total[path_of] > 0, seg / total[path_of] * extra, extra / (L - 1)[path_of])
    n = np.floor(share).astype(np.int64)
    # the points left over go to the largest remainders of each path, the first of equal ones first
    rest = W - L - np.bincount(path_of, weights=n, minlength=P).astype(np.int64)
    order = np.lexsort((n - share, path_of))
    rank = np.arange(path_of.size) - (first - np.arange(P))[path_of]
    n[order[rank < rest[path_of]]] += 1
    cnt = n + 1
    at = np.repeat(np.arange(path_of.size), cnt)                 # the segment of each point
    k = np.arange(at.size) - (np.cumsum(cnt) - cnt)[at]
    pts = v[a[at]] + (k / cnt[at])[:, None] * d[at]
    out = np.empty((P, W, v.shape[1]), np.float32)
    out[:, :-1] = pts.reshape(P, W - 1, -1)
    out[:, -1] = v[first + L - 1]
    return out


def _resample_paths(paths: list, W: int) -> np.ndarray:
    """resample_path of every path: [P, W, dim]."""
    paths = [np.asarray(p, dtype=np.float64) for p in paths]
    if all(p.ndim == 2 and 1 < p.shape[0] <= W and p.shape[1] == paths[0].shape[1] and np.isfinite(p).all() for p in paths):
        return _spread(paths, W)
    return np.stack([resample_path(p, W) for p in paths])


def densify(paths: torch.Tensor, resolution: float) -> tuple[torch.Tensor, torch.Tensor]:
    """Points every <= `resolution` (joint-space L2) along each polyline [P, W, dim];
    returns configs [M, dim] and the path index of each point."""
    P, W, dim = paths.shape
    dev = paths.device
    d = torch.linalg.norm(paths[:, 1:] - paths[:, :-1], dim=-1)           # [P, W-1]
    n = torch.clamp(torch.ceil(d / resolution), min=1).to(torch.int64)    # [P, W-1]
    # segment (p, w) gives points t = k / n for k < n, the last one also t = 1
    cnt = n.clone()
    cnt[:, -1] += 1
    cnt = cnt.reshape(-1)
    seg = torch.repeat_interleave(torch.arange(cnt.numel(), device=dev), cnt)
    first = torch.cumsum(cnt, 0) - cnt
    k = torch.arange(seg.numel(), device=dev) - first[seg]
    t = k.to(paths.dtype) / n.reshape(-1)[seg].to(paths.dtype)
    p, w = seg // (W - 1), seg % (W - 1)
    a, b = paths[p, w], paths[p, w + 1]
    return a + t[:, None] * (b - a), p


def smooth_paths(paths: list, collision_context: dict, lower, upper, *, waypoints: int = 64, steps: int = 50,
                 lr: float = 0.05, margin: float = 0.02, beta: float = 50.0, w_len: float = 1.0,
                 resolution: float = 0.01, device=None):
    """Smooth each path (list of [L_i, dim] arrays) with projected gradient steps
    on the adjoint cost; re-validate at `resolution`; revert paths that fail.
    A path of at most `waypoints` vertices reverts to itself (resample_path keeps
    its vertices); for a longer one the reverted waypoints are its arc-length
    resampling, and `accepted` tells the caller to keep the original path.

    Returns (smoothed [P, waypoints, dim] tensor, accepted [P] bool tensor,
    cost before [P], cost after [P])."""
    dev = cuda_device(device)
    dim = int(np.asarray(paths[0]).shape[1])
    init = torch.from_numpy(_resample_paths(paths, waypoints)).to(dev)
    lo = as_tensor(lower, torch.float32, dev).reshape(1, 1, dim)
    hi = as_tensor(upper, torch.float32, dev).reshape(1, 1, dim)
    sctx = SmoothContext(collision_context, dim, margin, beta, w_len, dev)
    x = init.clone()
    mask = torch.ones_like(x)
    mask[:, 0] = 0.0
    mask[:, -1] = 0.0
    c0, _ = sctx.cost_grad(init, need_grad=False, ordered=True)
    for _ in range(steps):
        _, g = sctx.cost_grad(x, ordered=True)
        # normalised step per path keeps the update scale independent of the cost scale
        gn = torch.linalg.norm((g * mask).reshape(g.shape[0], -1), dim=1).clamp_min(1e-12)
        x = torch.minimum(torch.maximum(x - lr * (g * mask) / gn[:, None, None], lo), hi)
    c1, _ = sctx.cost_grad(x, need_grad=False, ordered=True)
    checker = CollisionChecker(collision_context, dim, "binary", 0.0, dev)
    pts, owner = densify(x, resolution)
    v = checker.check(pts).to(torch.int64)
    bad = torch.zeros((x.shape[0],), dtype=torch.int64, device=dev).index_add_(0, owner, v)
    accepted = bad == 0
    out = torch.where(accepted[:, None, None], x, init)
    return out, accepted, c0, c1


class _BatchScenes:
    """Robot tables plus one world per problem, on the device in one staged
    copy, as the C struct of the batched entry points.  ``wait``: until that copy
    has run, for tables that are read on other streams than the current one."""

    def __init__(self, collision_contexts, device: torch.device, wait: bool = False):
        from .prrtc import _native_pack, _pack_worlds

        ctxs = list(collision_contexts)
        B = self.B = len(ctxs)
        # whether every context is the first one's robot in another world (the
        # very same tables), and none has a point cloud; a context of None is a
        # path without a world, which only the per-path check takes
        self.one_robot = all(c is not None and c.get("point_cloud") is None
                             and all(c.get(k) is ctxs[0].get(k) for k in ROBOT_SPEC) for c in ctxs)
        stage = Stager(device)
        self.robot_ctx = DeviceContext(ctxs[0], device, world_keys=False, stager=stage)
        native = _native_pack(ctxs, stage)
        if native is not None:
            keys = native[0]
        else:
            packed, counts = _pack_worlds(ctxs, B)
            keys = {k: (stage.add(packed[k], torch.int32 if k == "self_pairs" else torch.float32),
                        stage.add(counts[k], torch.int32), int(packed[k].shape[1])) for k in packed}
        stage.commit(wait=wait)
        self.robot_ctx.finish()
        self.stage = stage  # holds the tables
        bi = _lib.BatchInputs()
        bi.batch = B
        bi.robot = self.robot_ctx.robot()
        for key, (k_tab, k_cnt, width) in keys.items():
            setattr(bi, key, stage.address(k_tab))
            setattr(bi, "max_" + key, width)
            setattr(bi, key + "_count", stage.address(k_cnt) if k_cnt is not None else None)
        self.bi = bi


class BatchSmoothContext:
    """Robot tables plus one world per path, resident on the device, for the
    batched adjoint (prrtc_b200_smooth_cost_grad_batch): path p is costed
    against collision_contexts[p]'s world and self pairs.  The tables are on the
    device when the constructor returns, whatever stream reads them; with
    ``wait=False`` their copy is only queued, for use on the current stream."""

    def __init__(self, collision_contexts, dim: int, margin: float = 0.02, beta: float = 50.0, w_len: float = 1.0,
                 device=None, *, wait: bool = True):
        self.lib = _lib.load()
        self.device = cuda_device(device)
        self.dim = int(dim)
        self.margin, self.beta, self.w_len = float(margin), float(beta), float(w_len)
        self.scenes = _BatchScenes(collision_contexts, self.device, wait)
        self.B, self.bi = self.scenes.B, self.scenes.bi
        self.ws = workspace(self.lib.prrtc_b200_smooth_batch_workspace_size(C.byref(self.bi)), self.device)

    def cost_grad(self, waypoints: torch.Tensor, need_grad: bool = True, ordered: bool = True):
        """cost [P] and gradient [P, W, dim], the sums always in a fixed order."""
        wp = waypoints.detach().to(self.device, torch.float32).contiguous()
        P, W, dim = wp.shape
        if P != self.B:
            raise ValueError(f"expected {self.B} paths (one per world), got {P}")
        cost = torch.empty((P,), dtype=torch.float32, device=self.device)
        grad = torch.empty_like(wp) if need_grad else None
        _lib.check(self.lib.prrtc_b200_smooth_cost_grad_batch(C.byref(self.bi), dim, ptr(wp), W, self.margin,
                                                              self.beta, self.w_len, ptr(cost), ptr(grad),
                                                              self.ws.data_ptr(), self.ws.numel(), stream_handle()),
                   "prrtc_b200_smooth_cost_grad_batch")
        return cost, grad


    def descend(self, x: torch.Tensor, lo: torch.Tensor, hi: torch.Tensor, steps: int, lr: float) -> None:
        """`steps` projected gradient steps on x [P, W, dim] in place: per step the
        gradient (zero at the end points), its length per path, the update.
        The scenes are packed once."""
        P, W, dim = x.shape
        if P != self.B:
            raise ValueError(f"expected {self.B} paths (one per world), got {P}")
        g = torch.empty_like(x)
        lo, hi = (t.reshape(-1).expand(dim).contiguous() for t in (lo, hi))
        sp = stream_handle()
        for k in range(steps):
            _lib.check(self.lib.prrtc_b200_smooth_step_grad_batch(
                C.byref(self.bi), dim, x.data_ptr(), W, self.margin, self.beta, self.w_len, 1 if k else 0, g.data_ptr(),
                self.ws.data_ptr(), self.ws.numel(), sp), "prrtc_b200_smooth_step_grad_batch")
            norms = torch.linalg.norm(g.reshape(P, -1), dim=1)
            _lib.check(self.lib.prrtc_b200_smooth_update(x.data_ptr(), g.data_ptr(), norms.data_ptr(), lo.data_ptr(),
                                                         hi.data_ptr(), lr, P, W, dim, sp), "prrtc_b200_smooth_update")


def _differentiated(t: torch.Tensor) -> bool:
    return t.requires_grad or forward_ad.unpack_dual(t).tangent is not None


def projected_steps(sctx, init: torch.Tensor, lower, upper, steps: int, lr: float) -> torch.Tensor:
    """`steps` projected gradient steps of the adjoint cost from `init` [P, W, dim]:
    endpoints fixed, joint limits enforced, step length lr per path (the
    gradient normalised per path)."""
    P, W, dim = init.shape
    lo = as_tensor(lower, torch.float32, init.device).reshape(1, 1, dim)
    hi = as_tensor(upper, torch.float32, init.device).reshape(1, 1, dim)
    x = init.clone()
    # the kernels take plain memory of the scenes' device and one number for lr;
    # anything else (paths elsewhere, recorded by autograd or with tangents, without
    # an inner waypoint, another object's gradient) goes by the tensor expression
    if (isinstance(sctx, BatchSmoothContext) and type(sctx).cost_grad is BatchSmoothContext.cost_grad
            and type(x) is torch.Tensor and x.device == sctx.device and x.dtype == torch.float32 and x.is_contiguous()
            and P > 0 and W > 2 and isinstance(lr, (int, float)) and not any(map(_differentiated, (x, lo, hi)))):
        sctx.descend(x, lo, hi, steps, lr)
        return x
    order = {"ordered": True} if type(sctx) is SmoothContext else {}
    mask = torch.ones_like(x)
    mask[:, 0] = 0.0
    mask[:, -1] = 0.0
    for _ in range(steps):
        _, g = sctx.cost_grad(x, **order)
        gn = torch.linalg.norm((g * mask).reshape(P, -1), dim=1).clamp_min(1e-12)
        x = torch.minimum(torch.maximum(x - lr * (g * mask) / gn[:, None, None], lo), hi)
    return x


def smooth_paths_batch(paths: list, collision_contexts: list, lower, upper, *, waypoints: int = 64,
                       steps: int = 50, lr: float = 0.05, margin: float = 0.02, beta: float = 50.0,
                       w_len: float = 1.0, resolution: float = 0.01, device=None):
    """smooth_paths for the paths of a batch plan, path p in its own world
    collision_contexts[p]: one batched adjoint launch per step for all paths,
    then exact re-validation of each smoothed path at `resolution` against its
    world; a path that fails reverts to its input.

    Returns (smoothed [P, waypoints, dim], accepted [P] bool, cost before [P],
    cost after [P])."""
    dev = cuda_device(device)
    dim = int(np.asarray(paths[0]).shape[1])
    init = torch.from_numpy(_resample_paths(paths, waypoints)).to(dev)
    # used on this stream alone, and gone with the call
    sctx = BatchSmoothContext(collision_contexts, dim, margin, beta, w_len, dev, wait=False)
    c0, _ = sctx.cost_grad(init, need_grad=False)
    x = projected_steps(sctx, init, lower, upper, steps, lr)
    c1, _ = sctx.cost_grad(x, need_grad=False)
    accepted = revalidate_batch(x, collision_contexts, resolution, dev, sctx.scenes)
    out = torch.where(accepted[:, None, None], x, init)
    return out, accepted, c0, c1


def revalidate_batch(paths: torch.Tensor, collision_contexts: list, resolution: float, device,
                     scenes: _BatchScenes | None = None) -> torch.Tensor:
    """Exact binary re-validation of path p [W, dim] of `paths` at `resolution`
    against collision_contexts[p]; returns accepted [P] bool.  One batched
    check for all paths where their contexts are one robot in different worlds
    (``scenes``: their tables, when already on the device)."""
    pts, owner = densify(paths, resolution)
    P, dim = int(paths.shape[0]), int(paths.shape[2])
    dev = torch.empty(0, device=device).device  # None: torch's default
    lib = _lib.load()
    if P and pts.dtype == torch.float32 and pts.is_cuda:
        scenes = scenes if scenes is not None else _BatchScenes(collision_contexts, pts.device)
        if scenes.one_robot and scenes.B == P:
            offsets = torch.searchsorted(owner, torch.arange(P + 1, device=owner.device), out_int32=True)
            pts = pts.contiguous()
            v = torch.empty((pts.shape[0],), dtype=torch.int32, device=pts.device)
            ws = workspace(lib.prrtc_b200_check_configs_batch_workspace_size(C.byref(scenes.bi)), pts.device)
            rc = lib.prrtc_b200_check_configs_batch(C.byref(scenes.bi), dim, ptr(pts), ptr(offsets), int(pts.shape[0]),
                                                    0, 0.0, ptr(v), ws.data_ptr(), ws.numel(), stream_handle())
            if rc != _lib.EUNSUPPORTED:
                _lib.check(rc, "prrtc_b200_check_configs_batch")
                bad = torch.zeros((P,), dtype=torch.int32, device=pts.device).index_add_(0, owner, v)
                return (bad == 0).to(dev)
    owner_np = owner.cpu().numpy()
    bounds = np.searchsorted(owner_np, np.arange(paths.shape[0] + 1))
    accepted = torch.ones((paths.shape[0],), dtype=torch.bool, device=device)
    for p, ctx in enumerate(collision_contexts):
        seg = pts[bounds[p]:bounds[p + 1]]
        if seg.shape[0]:
            v = CollisionChecker(ctx, paths.shape[2], "binary", 0.0, device).check(seg)
            accepted[p] = v.max() == 0
    return accepted
