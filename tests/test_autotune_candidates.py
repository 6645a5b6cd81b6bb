"""What the autotuner times: no launch twice, and the explorer size that a launch of few explorers chooses among them."""
from __future__ import annotations

import types

import numpy as np
import pytest

from prrtc_b200 import autotune, scenes
from prrtc_b200.batch import PlanSettings
from prrtc_b200.context import build_collision_context


@pytest.mark.parametrize("coarse,problems", [(True, 512), (True, 61), (True, 4), (False, 61)])
def test_candidates_differ(coarse, problems):
    ctx = build_collision_context(scenes.arm(0), scenes.spheres_world(np.random.default_rng(0), 4))
    if not coarse:
        ctx = {**ctx, "fine_link_offsets": ctx["fine_link_offsets"][:0]}
    ps = [types.SimpleNamespace(context=ctx, dim=7)] * problems
    sms = 148
    cands = autotune._candidates(ps, PlanSettings(), sms)

    def launch(e, t, c, r):  # what reaches the device
        own = 512 if e * problems <= 2 * sms else 256
        return (e, (t or own) if coarse else (t or 128), None if coarse else c, r)

    assert len({launch(*c) for c in cands}) == len(cands)
    assert {e for e, *_ in cands} == set(autotune.SAMPLES) and {r for *_, r in cands} == set(autotune.CTAS_PER_SM)
    assert {t for _, t, *_ in cands} >= set(autotune.THREADS)
    assert {e for e, t, *_ in cands if t == 0} == ({e for e in autotune.SAMPLES if e * problems <= 2 * sms} if coarse else set())
    assert {c for *_, c, _ in cands} == (set(autotune.CHUNKS) if not coarse else {PlanSettings().waypoint_chunk})
