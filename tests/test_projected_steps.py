"""Which descents of projected_steps may go to the kernels: only plain memory of the scenes' own device.  Everything
else takes the tensor expression, with any object that has a cost_grad (CPU: the kernels' entry is replaced)."""
from __future__ import annotations

import numpy as np
import pytest
import torch

from prrtc_b200.smoothing import BatchSmoothContext, projected_steps


def _batch_context(device):
    """A BatchSmoothContext with tables on `device` (none here), a quadratic cost and a descend that records calls."""
    class Quadratic(BatchSmoothContext):
        def __init__(self):
            self.B, self.device, self.calls = 2, torch.device(device), []

        def descend(self, x, lo, hi, steps, lr):
            self.calls.append(x)

    s = Quadratic()
    return s


def _expected(init, lo, hi, steps, lr, grad):
    x = init.clone()
    mask = torch.ones_like(x)
    mask[:, 0] = mask[:, -1] = 0.0
    for _ in range(steps):
        g = grad(x) * mask
        x = torch.minimum(torch.maximum(x - lr * g / torch.linalg.norm(g.reshape(len(x), -1), dim=1).clamp_min(1e-12)[:, None, None],
                                        lo), hi)
    return x


@pytest.mark.parametrize("form", ["host_paths", "recorded", "strided", "float64", "two_waypoints", "tensor_lr", "limits_recorded"])
def test_kernels_take_plain_paths_only(form, monkeypatch):
    monkeypatch.setattr(BatchSmoothContext, "cost_grad", lambda self, x, need_grad=True: (None, 2.0 * x.detach()))
    s = _batch_context("cuda:0" if form == "host_paths" else "cpu")
    init = torch.from_numpy(np.random.default_rng(0).uniform(-1, 1, (2, 2 if form == "two_waypoints" else 6, 3)).astype(np.float32))
    if form == "recorded":
        init.requires_grad_(True)
    if form == "strided":
        init = init.transpose(1, 2).contiguous().transpose(1, 2)
    if form == "float64":
        init = init.double()
    lr = torch.tensor([0.1, 0.2])[:, None, None] if form == "tensor_lr" else 0.1
    lower = torch.full((3,), -0.9, requires_grad=form == "limits_recorded")
    x = projected_steps(s, init, lower, [0.9] * 3, 4, lr)
    assert not s.calls
    want = _expected(init, lower.reshape(1, 1, 3), torch.full((1, 1, 3), 0.9), 4, lr, lambda x: 2.0 * x.detach())
    assert torch.equal(x, want) and x.requires_grad == want.requires_grad
    if form == "recorded":
        assert torch.equal(torch.autograd.grad(x.sum(), init)[0], torch.autograd.grad(want.sum(), init)[0])


def test_tangents_are_kept(monkeypatch):
    """Paths in forward mode, inside the limits: the tangents come back with them (after no steps, as they went in)."""
    from torch.autograd import forward_ad

    monkeypatch.setattr(BatchSmoothContext, "cost_grad", lambda self, x, need_grad=True: (None, 2.0 * x.detach()))
    s = _batch_context("cpu")
    init, t = (torch.from_numpy(np.random.default_rng(k).uniform(-1, 1, (2, 6, 3)).astype(np.float32)) for k in (0, 1))
    with forward_ad.dual_level():
        x = projected_steps(s, forward_ad.make_dual(init, t), [-2.0] * 3, [2.0] * 3, 0, 0.1)
        assert not s.calls and torch.equal(forward_ad.unpack_dual(x).tangent, t)


def test_kernels_take_plain_paths(monkeypatch):
    monkeypatch.setattr(BatchSmoothContext, "cost_grad", lambda self, x, need_grad=True: (None, 2.0 * x))
    s = _batch_context("cpu")
    x = projected_steps(s, torch.zeros(2, 6, 3), [-1.0] * 3, [1.0] * 3, 4, 0.1)
    assert len(s.calls) == 1 and s.calls[0] is x


def test_own_cost_is_used():
    """An object of the caller's own, and a subclass with its own cost_grad."""
    class Own:
        def cost_grad(self, x):
            return None, 2.0 * x

    class Sub(BatchSmoothContext):
        def __init__(self):
            self.device, self.B = torch.device("cpu"), 2

        def cost_grad(self, waypoints, need_grad=True):
            return None, 2.0 * waypoints

    init = torch.from_numpy(np.random.default_rng(1).uniform(-1, 1, (2, 5, 3)).astype(np.float32))
    want = _expected(init, torch.tensor(-2.0), torch.tensor(2.0), 3, 0.1, lambda x: 2.0 * x)
    for sctx in (Own(), Sub()):
        assert torch.equal(projected_steps(sctx, init, [-2.0] * 3, [2.0] * 3, 3, 0.1), want)
