"""Scenes whose tables come to the last bytes of a CTA's shared memory (GPU): every count of world spheres around the
sizes where a kernel stops staging the scene is answered, by whichever form holds it.  Two spheres are 64 bytes."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest
import torch

from prrtc_b200 import scenes
from prrtc_b200.context import build_collision_context, with_world

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("call", ["check", "full_sweep", "gated", "smooth", "smooth_ordered"])
def test_every_scene_size(cuda, call):
    from prrtc_b200 import _lib
    from prrtc_b200.device import DeviceContext, stream_handle, workspace

    lib = _lib.load()
    robot = scenes.arm(0)
    most = 7600  # 243 KB: more than shared memory
    far = np.tile(np.array([[40.0, 0.0, 0.0, 0.1]], np.float32), (most, 1))
    tables = DeviceContext(with_world(build_collision_context(robot, None), {"world_spheres": far}), cuda)
    model, world = tables.robot(), tables.world()
    ws = workspace(max(lib.prrtc_b200_check_configs_workspace_size(C.byref(model), C.byref(world)),
                       lib.prrtc_b200_smooth_workspace_size(C.byref(model), C.byref(world))), cuda)
    q = torch.from_numpy(np.random.default_rng(0).uniform(-1, 1, (2, 4, robot.dim)).astype(np.float32)).to(cuda)
    cost, grad, hit = torch.empty(2, device=cuda), torch.empty_like(q), torch.empty(8, dtype=torch.int32, device=cuda)
    seen = []
    for n in range(1000, most + 1, 2):
        world.n_world_spheres = n
        if call.startswith("smooth"):
            entry = lib.prrtc_b200_smooth_cost_grad if call == "smooth" else lib.prrtc_b200_smooth_cost_grad_ordered
            rc = entry(C.byref(model), C.byref(world), robot.dim, q.data_ptr(), 2, 4, 0.02, 50.0, 1.0, cost.data_ptr(),
                       grad.data_ptr(), ws.data_ptr(), ws.numel(), stream_handle())
            out = grad
        else:
            rc = lib.prrtc_b200_check_configs(C.byref(model), C.byref(world), robot.dim, q.data_ptr(), 8, 2 if call == "gated" else 0,
                                              0.0, int(call == "full_sweep"), hit.data_ptr(), ws.data_ptr(), ws.numel(), stream_handle())
            out = hit
        assert rc == 0, (n, rc)
        if n % 300 == 0:
            seen.append(out.clone())
    # far spheres change nothing but the order of sums in the forms that take a lane per waypoint
    for out in seen[1:]:
        assert torch.equal(out, seen[0]) if call != "smooth" else torch.allclose(out, seen[0], rtol=0, atol=1e-3 * float(seen[0].abs().max()))
