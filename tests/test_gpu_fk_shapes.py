"""Forward kinematics at the edges of the kernel's tile (GPU): one joint to the largest table, configuration counts
around a tile of 40 and above one pass of the grid, branching parents, permuted output frames, an output that is not
16-byte aligned.  Compared with the oracle's float64 frames."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest
import torch

from prrtc_b200 import scenes

pytestmark = pytest.mark.gpu

OFFSET = 0.1  # each joint's offset from its parent, at most


def _tables(J: int, dim: int, seed: int) -> dict:
    rng = np.random.default_rng(seed)
    rob = scenes.arm(0, 7)
    sel = np.arange(J) % 7
    ptf = np.array(rob.parent_tf, np.float32)[sel]
    ptf[:, 4:7] = rng.uniform(-1, 1, (J, 3)) * OFFSET / np.sqrt(3)
    parent = np.array([int(rng.integers(max(0, j - 3), j)) if j and j % 11 else -1 for j in range(J)], np.int32)
    return {"fk_twists": np.array(rob.twists, np.float32)[sel], "fk_parent_tf": ptf, "fk_parent_idx": parent,
            "fk_act_idx": (np.arange(J) % dim).astype(np.int32), "fk_mimic_mul": np.ones(J, np.float32),
            "fk_mimic_off": np.zeros(J, np.float32), "fk_mimic_act_idx": np.full(J, -1, np.int32),
            "fk_topo_inv": rng.permutation(J).astype(np.int32)}


@pytest.mark.parametrize("shift", [0, 1])  # floats between the output and a 16-byte boundary
@pytest.mark.parametrize("J,dim,n", [(1, 1, 1), (7, 7, 39), (7, 7, 40), (18, 14, 41), (33, 16, 121), (64, 16, 81),
                                     (3, 2, 8 * 160 * 40 + 1)])
def test_shapes(cuda, orc, J, dim, n, shift):
    from prrtc_b200 import _lib
    from prrtc_b200.device import DeviceContext, stream_handle

    ctx = _tables(J, dim, J)
    q = np.random.default_rng(n).uniform(-2.8, 2.8, (n, dim)).astype(np.float32)
    qd = torch.from_numpy(q).to(cuda)
    buf = torch.full((n * J * 12 + 8,), 7.0, device=cuda)
    dc = DeviceContext(ctx, cuda, world_keys=False)
    robot = dc.robot()
    _lib.check(_lib.load().prrtc_b200_fk(C.byref(robot), dim, qd.data_ptr(), n, buf[shift:].data_ptr(),
                                         stream_handle()), "prrtc_b200_fk")
    out = buf.cpu().numpy()
    assert np.all(out[:shift] == 7.0) and np.all(out[shift + n * J * 12:] == 7.0)
    F = out[shift:shift + n * J * 12].reshape(n, J, 12)
    # a composition rounds to about 8 units in the last place of 1 + reach, once per joint of the chain
    tol = 8 * 2.0**-24 * J * (1 + J * OFFSET)
    sc = orc.Scene(ctx, dim)
    for i in sorted({0, 1, n // 2, n - 2, n - 1, *range(37, 43)} & set(range(n))):
        assert np.abs(F[i] - sc.fk(q[i].astype(np.float64))).max() <= tol
