"""A call that finds no memory for its workspace returns an error and leaves the
context usable: the next, smaller call allocates what it needs."""
from __future__ import annotations

import numpy as np
import pytest

import horender as hr
import mlp_ref

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def test_gradients_after_a_failed_allocation():
    ctx, _ = hr.workload_context("hex4_p4")
    ctx.mlp_init(6)
    rng = np.random.default_rng(1)
    X = rng.normal(size=(64, 48)).astype(np.float32)
    T = rng.normal(size=(64, 8)).astype(np.float32)
    ok = np.ones(64, np.uint8)
    n = 1 << 20  # 0.24 GB of rows fit beside the block below, their 1.8 GB of activations do not
    big = np.zeros((n, 48), np.float32), np.zeros((n, 8), np.float32), np.ones(n, np.uint8)
    ctx.mlp_grad(X[:8], T[:8], ok[:8])
    torch.cuda.synchronize()
    free, _ = torch.cuda.mem_get_info()
    block = torch.empty(free - (1 << 30), dtype=torch.uint8, device="cuda")
    try:
        with pytest.raises(hr.HoError):
            ctx.mlp_grad(*big)
        loss, g = ctx.mlp_grad(X, T, ok)
    finally:
        del block
        torch.cuda.empty_cache()
    rloss, rg = mlp_ref.loss_and_grads(ctx.mlp_params(), X, T, ok)
    assert abs(loss - rloss) <= 1e-3 * rloss
    assert np.linalg.norm(g - rg) <= 3e-2 * np.linalg.norm(rg)
