"""Resampling of many paths at once: the same bits as a path at a time, for every vertex count up to the waypoints, equal
segments (ties among the remainders), repeated vertices, paths without length and batches that fall back."""
from __future__ import annotations

import numpy as np
import pytest

from prrtc_b200.smoothing import _resample_paths, resample_path


@pytest.mark.parametrize("W,dim,P", [(2, 7, 1), (3, 1, 5), (16, 7, 9), (64, 7, 32), (65, 14, 4), (33, 16, 3)])
@pytest.mark.parametrize("form", ["plain", "equal", "repeated", "point", "mixed", "not_finite"])
def test_matches_one_path_at_a_time(W, dim, P, form):
    rng = np.random.default_rng(W * 100 + dim)
    paths = []
    for p in range(P):
        L = int(rng.integers(2, W + 1)) if form != "mixed" else int(rng.integers(1, W + 5))
        x = rng.uniform(-2.8, 2.8, (L, dim))
        if form == "equal":
            x = np.arange(L)[:, None] * np.full((1, dim), 0.5)
        elif form == "repeated":
            x = x[np.arange(L) // 2]
        elif form == "point":
            x[:] = 0.25
        elif form == "not_finite" and p == 0:
            x[-1, 0] = np.nan
        paths.append(x.astype(np.float32) if p % 2 else x)
    with np.errstate(invalid="ignore"):
        try:
            want = np.stack([resample_path(p, W) for p in paths])
        except ValueError:
            with pytest.raises(ValueError):
                _resample_paths(paths, W)
            return
        got = _resample_paths(paths, W)
    assert got.dtype == want.dtype and np.array_equal(got.view(np.uint32), want.view(np.uint32))
