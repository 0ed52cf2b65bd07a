"""The engine on elements with a convergence certificate (excluded isosurface
searches, staged seeds, short face slots): scenes in which all, some or none of
the elements have one, at the orders where a face batch holds 32 slots (up to 7
modes a direction), 22 (8 modes) and 14 (9 modes). Which elements have one is
read back, so that a scene which no longer has them fails here."""
from __future__ import annotations

import numpy as np
import pytest

import horender as hr
import parity
from conftest import scene_arrays_from_ctx

pytestmark = pytest.mark.gpu

# elements a side, order, curving amplitude over the element size; which certified
SCENES = {
    "none": (5, 6, 0.05), "all": (16, 6, 0.02), "some": (20, 6, 0.08),
    "some-order2": (24, 2, 0.08), "some-order7": (16, 7, 0.05), "some-order8": (16, 8, 0.05),
}


@pytest.fixture(scope="module", params=SCENES.items(), ids=list(SCENES))
def scene(request):
    label, (side, order, amp) = request.param
    ctx = hr.Context(0)
    ctx.generate_synthetic(side, side, side, order, order, amp, 24, 7)
    assert ctx.get_option(hr.OPT_CERTIFIED) == 0  # not built yet
    ctx.build_bvh()
    n = ctx.get_option(hr.OPT_CERTIFIED)
    want = {"none": n == 0, "all": n == side ** 3, "some": side ** 3 // 4 < n < side ** 3}
    assert want[label.split("-")[0]], (label, n)
    yield label, ctx, side
    ctx.close()


def some_rays(n, seed):
    rng = np.random.default_rng(seed)
    o = rng.uniform(-0.4, 1.4, (n, 3))
    d = rng.uniform(0.05, 0.95, (n, 3)) - o
    return np.concatenate([o, d / np.linalg.norm(d, axis=1, keepdims=True)], 1).astype(np.float32)


def isovalues(ctx, rays):
    """Just inside the largest and in the middle of the field's face values."""
    u = ctx.intersect(rays, 0.0, False)["u"]
    return float(u.max()) - 1e-3, float(np.median(u))


@pytest.mark.parametrize("tail", [0, 4])
def test_batch_sizes_change_no_answer(scene, tail):
    label, ctx, side = scene
    rays = some_rays(40_000, 1)
    iso = isovalues(ctx, rays)[1]
    unset = ctx.get_option(hr.OPT_ROUND_CHUNK)
    try:
        ctx.set_option(hr.OPT_TAIL, tail)
        a = ctx.intersect(rays, iso, True)
        assert ctx.stats()["status"] == 0 and (a["kind"] == hr.HIT_FACE).any() and (a["kind"] == hr.HIT_ISO).any()
        for chunk in (3, 32, 100):
            ctx.set_option(hr.OPT_ROUND_CHUNK, chunk)
            b = ctx.intersect(rays, iso, True)
            for k in ("t", "elem", "face", "kind", "xi", "n", "u", "flags"):
                assert np.array_equal(a[k], b[k]), (label, k, chunk)
    finally:
        ctx.set_option(hr.OPT_ROUND_CHUNK, unset)
        ctx.set_option(hr.OPT_TAIL, 4)


def test_against_64_bits(scene, oracle):
    label, ctx, side = scene
    osc = oracle.OracleScene(scene_arrays_from_ctx(ctx))
    rays = some_rays(2500, 3)
    for iso in isovalues(ctx, rays):
        h = ctx.intersect(rays, iso, True)
        parity.check_against_oracle(h, rays, osc, iso, True, 1.0 / side,
                                    product_trace=lambda r: ctx.intersect(r, iso, True),
                                    label=f"{label}, isovalue {iso:.3f}")
