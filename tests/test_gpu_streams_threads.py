"""Objects used on another stream than the one they were made on, and calls from several host threads (GPU)."""
from __future__ import annotations

import ctypes as C
import threading

import numpy as np
import pytest
import torch

from prrtc_b200 import scenes
from prrtc_b200.context import build_collision_context, with_world

pytestmark = pytest.mark.gpu


def _paths(robot, P, W, seed, device):
    q = np.random.default_rng(seed).uniform(-1.0, 1.0, (P, W, robot.dim)).astype(np.float32)
    return torch.from_numpy(q).to(device)


def test_batch_smoothing_context_on_another_stream(cuda):
    """Built on a stream with work in front, evaluated at once on another stream: the tables have to be there."""
    from prrtc_b200.smoothing import BatchSmoothContext

    robot = scenes.arm(0)
    base = build_collision_context(robot, None)
    ctxs = [with_world(base, scenes.tabletop_world(np.random.default_rng(k))) for k in range(5)]
    x = _paths(robot, 5, 17, 3, cuda)
    cost, grad = BatchSmoothContext(ctxs, robot.dim, device=cuda).cost_grad(x)
    torch.cuda.synchronize()
    one, other = torch.cuda.Stream(cuda), torch.cuda.Stream(cuda)
    with torch.cuda.stream(one):
        torch.cuda._sleep(100_000_000)  # about 50 ms
        sctx = BatchSmoothContext(ctxs, robot.dim, device=cuda)
    with torch.cuda.stream(other):
        got_cost, got_grad = sctx.cost_grad(x)
    torch.cuda.synchronize()
    # the sums of a gradient have one order; a path's cost is added up over its waypoints in any order (17 terms of one
    # sign: 16 roundings of 2^-24 each)
    assert torch.equal(got_grad, grad)
    assert torch.allclose(got_cost, cost, rtol=2e-6, atol=0.0)


@pytest.mark.parametrize("what", ["one_scene", "ordered", "scene_per_path", "frames"])
def test_two_threads_with_tables_of_different_sizes(cuda, what):
    """The shared memory that a launch asks for grows with the scene (smoothing) or the joints (frames): one thread's
    small call must not lower the limit under the other's large one.  Plain calls of the C entries, one after the other,
    on a stream per thread; each call has to go through and the last result of a thread to be the one of a call alone."""
    from prrtc_b200 import _lib
    from prrtc_b200.device import DeviceContext
    from prrtc_b200.smoothing import BatchSmoothContext, SmoothContext
    from test_gpu_fk_shapes import _tables

    lib = _lib.load()
    robot = scenes.arm(0)
    base = build_collision_context(robot, None)
    worlds = [with_world(base, scenes.spheres_world(np.random.default_rng(5), n)) for n in (16, 1500)]
    x = _paths(robot, 2, 2, 1, cuda)
    if what == "frames":
        ctx = [DeviceContext(_tables(J, 7, J), cuda, world_keys=False) for J in (30, 64)]
        robots = [c.robot() for c in ctx]
        out = [torch.zeros(4 * J * 12, device=cuda) for J in (30, 64)]
        call = lambda k, s: lib.prrtc_b200_fk(C.byref(robots[k]), 7, x.data_ptr(), 4, out[k].data_ptr(), s)  # noqa: E731
    else:
        cost = [torch.zeros(2, device=cuda) for _ in worlds]
        out = [torch.zeros_like(x) for _ in worlds]
        tail = lambda k, s: (cost[k].data_ptr(), out[k].data_ptr(), ctx[k].ws.data_ptr(), ctx[k].ws.numel(), s)  # noqa: E731
        if what == "scene_per_path":
            ctx = [BatchSmoothContext([w, w], robot.dim, device=cuda) for w in worlds]
            call = lambda k, s: lib.prrtc_b200_smooth_cost_grad_batch(  # noqa: E731
                C.byref(ctx[k].bi), 7, x.data_ptr(), 2, 0.02, 50.0, 1.0, *tail(k, s))
        else:
            ctx = [SmoothContext(w, robot.dim, device=cuda) for w in worlds]
            entry = lib.prrtc_b200_smooth_cost_grad_ordered if what == "ordered" else lib.prrtc_b200_smooth_cost_grad
            call = lambda k, s: entry(C.byref(ctx[k].robot), C.byref(ctx[k].world), 7, x.data_ptr(), 2, 2, 0.02, 50.0,  # noqa: E731
                                      1.0, *tail(k, s))
    want = []
    for k in (0, 1):
        _lib.check(call(k, torch.cuda.current_stream().cuda_stream), what)
        torch.cuda.synchronize()
        want.append(out[k].clone())
    codes, gate = [[], []], threading.Barrier(2)

    def work(k):
        torch.cuda.set_device(cuda)
        stream = torch.cuda.Stream(cuda)
        gate.wait()
        for n in range(4000):
            codes[k].append(call(k, stream.cuda_stream))
            if n % 200 == 199:
                stream.synchronize()

    threads = [threading.Thread(target=work, args=(k,)) for k in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join(120)
    torch.cuda.synchronize()
    assert [len(c) for c in codes] == [4000, 4000] and not any(codes[0]) and not any(codes[1])
    for k in (0, 1):
        # one scene's sums may be taken in any order: a sum of about 2,000 terms, each rounded to 2^-24 of the largest
        assert torch.allclose(out[k], want[k], rtol=1e-4, atol=1e-4) if what == "one_scene" else torch.equal(out[k], want[k])
