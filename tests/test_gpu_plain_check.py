"""The plain mode's FP64 check sums a face hit over the face at some orders and
over the element at the others: at every order its hits are polished to exact
roots. The FP64 position residual of a polished hit is the rounding of t and xi
to FP32, at most half an ulp of t <= 4 (2.4e-7) and |J| of half an element times
half an ulp of 1 (3e-8) a coordinate: under 5e-7 on all but hits at which a
polish cannot help (off the face, near-tangent), which are under 1%."""
from __future__ import annotations

import numpy as np
import pytest

import horender as hr

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", range(1, 9))
def test_plain_hits_are_roots(order):
    ctx = hr.Context(0)
    ctx.generate_synthetic(4, 4, 4, order, order, 0.05, 16, 3)
    ctx.build_bvh()
    ctx.set_mode(hr.MODE_PLAIN)
    rng = np.random.default_rng(order)
    d = rng.normal(size=(3000, 3))
    o = rng.uniform(0.2, 0.8, (3000, 3)) - 1.5 * d / np.linalg.norm(d, axis=1, keepdims=True)
    rays = np.concatenate([o, d / np.linalg.norm(d, axis=1, keepdims=True)], 1).astype(np.float32)
    h = ctx.intersect(rays, 0.1, True)
    res = np.asarray(ctx.hit_residuals(rays, h)).reshape(-1, 2)[h["kind"] > 0, 0]
    assert (h["kind"] == hr.HIT_FACE).sum() > 300
    assert np.quantile(res, 0.99) < 5e-7, np.quantile(res, [0.5, 0.9, 0.99, 1.0])
