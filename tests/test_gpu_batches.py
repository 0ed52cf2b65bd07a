"""How many pairs share a batch of the round kernel depends on how many a round
has: the answers may not. Calls around the sizes where the rule changes (one pair
a batch, a few, full batches), against the same call with full batches set
explicitly, bit for bit."""
from __future__ import annotations

import numpy as np
import pytest

import horender as hr

pytestmark = pytest.mark.gpu


def scene(order, amp):
    c = hr.Context(0)
    c.generate_synthetic(5, 5, 5, order, order, amp, 32, 11)
    c.build_bvh()
    return c


@pytest.fixture(scope="module", params=[(3, 0.2), (6, 0.05)], ids=["uncertified", "certified"])
def pair(request):
    return scene(*request.param), scene(*request.param)


@pytest.mark.parametrize("n", [1, 33, 2500, 6000, 60000])
def test_batch_sizes_change_no_answer(pair, n):
    free, fixed = pair
    rng = np.random.default_rng(n)
    o = rng.uniform(-0.6, 1.6, (n, 3))
    d = rng.uniform(0.1, 0.9, (n, 3)) - o
    rays = np.concatenate([o, d / np.linalg.norm(d, axis=1, keepdims=True)], 1).astype(np.float32)
    a = free.intersect(rays, 0.1, True)
    for chunk in (7, 32):
        fixed.set_option(hr.OPT_ROUND_CHUNK, chunk)
        b = fixed.intersect(rays, 0.1, True)
        for k in ("t", "elem", "face", "kind", "xi", "n", "u", "flags"):
            assert np.array_equal(a[k], b[k]), (k, chunk)
