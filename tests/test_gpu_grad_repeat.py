"""A gradient call on the same rows gives the same bits every time: the loss and
the bias gradients at any size, the weight gradients below 1,024 rows (above,
the parts of their sums over the rows arrive in any order)."""
from __future__ import annotations

import numpy as np
import pytest

import horender as hr
import mlp_ref

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def net():
    c, _ = hr.workload_context("hex4_p4")
    c.mlp_init(3)
    return c


@pytest.mark.parametrize("n", [65, 512, 513, 1023, 6000])
def test_gradients_repeat(net, n):
    rng = np.random.default_rng(n)
    X = rng.normal(size=(n, 48)).astype(np.float32)
    T = rng.normal(size=(n, 8)).astype(np.float32)
    valid = (rng.uniform(size=n) > 0.1).astype(np.uint8)
    loss, g = net.mlp_grad(X, T, valid)
    for _ in range(10):
        loss2, g2 = net.mlp_grad(X, T, valid)
        assert loss2 == loss
        o = 0
        for i, m in mlp_ref.DIMS:
            if n < 1024:
                assert np.array_equal(g2[o:o + i * m], g[o:o + i * m]), o
            o += i * m
            assert np.array_equal(g2[o:o + m], g[o:o + m]), o
            o += m
