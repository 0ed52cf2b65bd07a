"""The batch size that HO_OPT_ROUND_CHUNK reports while unset stands for the
rule by each round's pairs: setting it (a program that puts an option back, the
autotuner) leaves small calls spread over the device. Counted in the warps'
solver steps: at one pair a batch, which a call of 777 rays gets by the rule,
they are the sum of the pairs' own chains, the same in every run, and full
batches take fewer."""
from __future__ import annotations

import numpy as np
import pytest

import horender as hr

pytestmark = pytest.mark.gpu


def test_reported_size_is_the_rule():
    ctx, w = hr.workload_context("hex4_p4")
    rng = np.random.default_rng(5)
    o = rng.uniform(-0.6, 1.6, (777, 3))
    d = rng.uniform(0.1, 0.9, (777, 3)) - o
    rays = np.concatenate([o, d / np.linalg.norm(d, axis=1, keepdims=True)], 1).astype(np.float32)

    def steps():
        ctx.intersect(rays, 0.2, True)
        return ctx.stats()["solve_steps"]

    unset = ctx.get_option(hr.OPT_ROUND_CHUNK)
    free = steps()
    assert steps() == free
    ctx.set_option(hr.OPT_ROUND_CHUNK, unset)
    assert steps() == free
    ctx.set_option(hr.OPT_ROUND_CHUNK, 2 * unset)
    assert steps() < free
    ctx.autotune(w.camera, w.isovalues, 64, 64)
    ctx.set_option(hr.OPT_ROUND_CHUNK, unset)
    assert steps() == free
