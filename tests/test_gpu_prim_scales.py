"""The primitive pass on directions that are not unit vectors, against the FP32
oracle, exactly: the bounds that leave a primitive out hold for every ray whose
answer the solvers can find, so also where a short direction goes with a large
t (prisms 100 units across and directions of 2e-19: the ray's rate along a
prism's bounds falls below 1e-20, its t to the far side is 5e20)."""
from __future__ import annotations

import numpy as np
import pytest

import horender as hr
import prim_synth as syn
from test_gpu_prims import compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("length", [2e-19, 1e-3, 1.0, 1e5])
@pytest.mark.parametrize("kind", [syn.PRISM, syn.QUAD, syn.TRI], ids=["prism", "quad", "tri"])
def test_direction_lengths(oracle, kind, length):
    rng = np.random.default_rng(3)
    b = syn.Builder()
    for _ in range(6):
        if kind == syn.PRISM:
            v = np.array(syn.tent(0, 0, 0, 60, 60, 40)) + rng.normal(size=(6, 3)) * 4
        elif kind == syn.QUAD:
            v = np.array([(0, 0, 0), (60, 0, 0), (0, 0, 60), (60, 0, 60)]) + rng.normal(size=(4, 3)) * 8
        else:
            v = np.array([(0, 0, 0), (60, 0, 0), (0, 60, 0)]) + rng.normal(size=(3, 3)) * 8
        b.add(kind, v + rng.uniform(0, 40, 3), None, (0, 0, 0), None, (0, 0, 0))
    arrs = b.build()
    o = rng.uniform(0, 100, (1500, 3))
    d = rng.uniform(0, 100, (1500, 3)) - o
    d *= length / np.linalg.norm(d, axis=1, keepdims=True)
    rays = np.concatenate([o, d], 1).astype(np.float32)
    ctx = hr.Context(0)
    ctx.add_prim_arrays(arrs)
    ctx.build_bvh()
    ref = oracle.OraclePrims(arrs).trace(rays, None, 32)
    compare(ctx.intersect(rays, 0.0, False), ref, f"{kind} {length}")
    if kind == syn.PRISM:
        assert (ref["kind"] > 0).any()
