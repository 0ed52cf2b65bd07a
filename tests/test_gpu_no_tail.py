"""Without a tail, a call runs as many rounds as the call before needed, and more
while rays are left. How many it starts with may not change an answer: the first
call after one that ran few rounds against a second one, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

import horender as hr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("side,order,amp", [(5, 6, 0.05), (16, 6, 0.02), (24, 2, 0.08)])
def test_call_does_not_depend_on_the_one_before(side, order, amp):
    ctx = hr.Context(0)
    ctx.generate_synthetic(side, side, side, order, order, amp, 24, 7)
    ctx.build_bvh()
    rng = np.random.default_rng(2)
    o = rng.uniform(-0.4, 1.4, (40_000, 3))
    d = rng.uniform(0.05, 0.95, o.shape) - o
    rays = np.concatenate([o, d / np.linalg.norm(d, axis=1, keepdims=True)], 1).astype(np.float32)
    ctx.set_option(hr.OPT_TAIL, 1)
    ctx.intersect(rays, 0.1, True)
    ctx.set_option(hr.OPT_TAIL, 0)
    a, first = ctx.intersect(rays, 0.1, True), ctx.stats()
    b, second = ctx.intersect(rays, 0.1, True), ctx.stats()
    assert first["rounds"] == second["rounds"] > 2
    for k in ("t", "elem", "face", "kind", "xi", "n", "u", "flags"):
        assert np.array_equal(a[k], b[k]), k
    # every hit is checked once
    assert first["fp64_checked"] == second["fp64_checked"] == (a["kind"] > 0).sum()
