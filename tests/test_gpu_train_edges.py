"""The training kernels at the edges of their tiles (32 rows a tile of the
forward and backward pass, 256 rows a chunk of the weight gradients, 32 chunks
side by side) against the float64 restatement, which rounds to BF16 at the same
points. Bounds as for the gradients at 512 rows: what differs is the FP32
accumulation, which now and then moves an activation to the next BF16 value
(2^-8 of it)."""
from __future__ import annotations

import numpy as np
import pytest

import horender as hr
import mlp_ref

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def net():
    c, _ = hr.workload_context("hex4_p4")
    c.mlp_init(6)
    return c


@pytest.mark.parametrize("n", [1, 31, 32, 33, 255, 256, 257, 4865, 8193, 16500])
def test_gradients_at_tile_edges(net, n):
    rng = np.random.default_rng(n)
    X = rng.normal(size=(n, 48)).astype(np.float32)
    T = rng.normal(size=(n, 8)).astype(np.float32)
    valid = (rng.uniform(size=n) > 0.2).astype(np.uint8)
    valid[-1] = 1
    loss, g = net.mlp_grad(X, T, valid)
    rloss, rg = mlp_ref.loss_and_grads(net.mlp_params(), X, T, valid)
    assert abs(loss - rloss) <= 1e-3 * rloss
    o = 0
    for i, nn in mlp_ref.DIMS:
        for size in (i * nn, nn):
            a, b = g[o:o + size], rg[o:o + size]
            assert np.linalg.norm(a - b) <= 3e-2 * max(np.linalg.norm(b), 1e-12), (n, o)
            o += size


def test_no_valid_row(net):
    loss, g = net.mlp_grad(np.ones((40, 48), np.float32), np.full((40, 8), np.nan, np.float32), np.zeros(40, np.uint8))
    assert loss == 0.0 and not g.any()
