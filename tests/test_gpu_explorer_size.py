"""The explorer size that a caller names is the one that runs; without one, few explorers get 512 threads (GPU: block
sizes as the profiler records them)."""
from __future__ import annotations

import json

import numpy as np
import pytest
import torch

from prrtc_b200 import scenes
from prrtc_b200.context import build_collision_context

pytestmark = pytest.mark.gpu


def _block(call, tmp_path):
    with torch.profiler.profile(activities=[torch.profiler.ProfilerActivity.CUDA]) as prof:
        call()
        torch.cuda.synchronize()
    path = tmp_path / "trace.json"
    prof.export_chrome_trace(str(path))
    ran = [e["args"]["block"][0] for e in json.loads(path.read_text())["traceEvents"]
           if "explore_kernel" in e.get("name", "") and "block" in e.get("args", {})]
    if not ran:
        pytest.skip("the profiler records no launches here")
    return set(ran)


@pytest.mark.parametrize("launch", ["persistent", "per_problem"])
def test_a_named_size_runs(cuda, tmp_path, launch):
    from prrtc_b200 import prrtc_plan_batch

    robot = scenes.arm(0)
    ctx = build_collision_context(robot, scenes.spheres_world(np.random.default_rng(3), 16))
    q = np.random.default_rng(4).uniform(-1.0, 1.0, (2, 5, robot.dim)).astype(np.float32)

    def plan(threads):
        return lambda: prrtc_plan_batch(q[0], q[1][:, None], collision_context=[ctx] * 5, launch=launch, max_iterations=20,
                                        num_new_samples=2, max_nodes=512, min_vals=robot.lower, max_vals=robot.upper,
                                        threads_per_explorer=threads)

    for threads in (64, 128, 256):
        assert _block(plan(threads), tmp_path) == {threads}
    assert _block(plan(0), tmp_path) == {512}
