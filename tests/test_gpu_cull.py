"""Candidates that end without a solve, at the edges of the rule: isovalues
just inside and outside the field's range, elements whose curving defeats the
certificate, the lowest and highest orders, rays that start inside the mesh.
Every difference from the FP64 oracle, which runs every search, must be one of
the classes of tests/parity.py, and the errors stay within its bounds."""
from __future__ import annotations

import numpy as np
import pytest

import horender as hr
import parity
from conftest import scene_arrays_from_ctx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order,amp", [(1, 0.05), (4, 0.15), (8, 0.1)])
def test_excluded_searches_change_no_answer(oracle, order, amp):
    ctx = hr.Context(0)
    ctx.generate_synthetic(5, 5, 5, order, order, amp, 16, 31 + order)
    ctx.build_bvh()
    osc = oracle.OracleScene(scene_arrays_from_ctx(ctx))
    rng = np.random.default_rng(order)
    n = 700
    o = rng.uniform(-0.3, 1.3, (n, 3))
    d = rng.normal(size=(n, 3))
    rays = np.concatenate([o, d / np.linalg.norm(d, axis=1, keepdims=True)], 1).astype(np.float32)
    u = ctx.intersect(rays, 0.0, False)["u"]  # field values on the elements' faces
    for iso in (float(u.min()) - 1e-3, float(u.max()) - 1e-3, float(np.median(u))):
        h = ctx.intersect(rays, iso, True)
        parity.check_against_oracle(h, rays, osc, iso, True, 0.2, product_trace=lambda r: ctx.intersect(r, iso, True),
                                    label=f"order {order}, isovalue {iso:.3f}")
