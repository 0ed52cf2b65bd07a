"""The primitive pass's searches against the FP32 oracle, exactly: orders with
an unrolled evaluation (2 to 5 modes, equal in all directions) and those beyond
it (6 modes, unequal modes, linear), rays that miss a primitive's bounds, graze
them or pass several primitives, and queries that run past the budget after
which a warp takes them over. The kernels run the reference's FP32 steps
without contraction, so nothing may differ: no tolerance."""
from __future__ import annotations

import numpy as np
import pytest

import horender as hr
import prim_synth as syn
from test_gpu_prims import compare

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def scene(kinds, modes, seed):
    rng = np.random.default_rng(seed)
    b = syn.Builder()
    for i in range(18):
        kind = kinds[i % len(kinds)]
        if kind == syn.PRISM:
            v = np.array(syn.tent(0, 0, 0, 0.3, 0.3, 0.2)) + rng.normal(size=(6, 3)) * 0.02
        elif kind == syn.QUAD:
            v = np.array([(0, 0, 0), (0.3, 0, 0), (0, 0, 0.3), (0.3, 0, 0.3)]) + rng.normal(size=(4, 3)) * 0.04
        else:
            v = np.array([(0, 0, 0), (0.3, 0, 0), (0, 0.3, 0)]) + rng.normal(size=(3, 3)) * 0.04
        v = v + rng.uniform(0, 0.7, 3)
        m = modes if kind == syn.PRISM else modes[:2] + (0,)
        linear = modes[0] == 0
        g = None if linear else syn.fit_geometry(kind, v, m, 0.04, rng.normal(size=3))
        b.add(kind, v, g, (0, 0, 0) if linear else m, None, (0, 0, 0))
    o = rng.uniform(-0.3, 1.4, (1500, 3))
    d = rng.uniform(0, 1, (1500, 3)) - o
    rays = np.concatenate([o, d / np.linalg.norm(d, axis=1, keepdims=True)], 1).astype(np.float32)
    rays[-3:, 3:] = [(0, 0, 1), (1, 0, 0), (0, -1, 0)]  # components below the slab test's limit
    return b.build(), rays


@pytest.mark.parametrize("kinds", [(syn.PRISM,), (syn.QUAD,), (syn.TRI,), (syn.PRISM, syn.QUAD, syn.TRI)],
                         ids=["prism", "quad", "tri", "all"])
@pytest.mark.parametrize("modes", [(0, 0, 0), (2, 2, 2), (4, 4, 4), (5, 5, 5), (6, 6, 6), (3, 4, 5)], ids=str)
def test_searches_match_oracle(oracle, kinds, modes):
    arrs, rays = scene(kinds, modes, 7 + modes[0] + 10 * kinds[0])
    ctx = hr.Context(0)
    ctx.add_prim_arrays(arrs)
    ctx.build_bvh()
    ref = oracle.OraclePrims(arrs).trace(rays, None, 32)
    n = rays.shape[0]
    dr = torch.from_numpy(rays).cuda()
    out = torch.zeros((3, n, 12), dtype=torch.int32, device="cuda")
    s = torch.cuda.Stream()
    # the forms that do not hand over: no allocation, and under capture
    ctx.intersect_device_noalloc(n, dr.data_ptr(), 0.0, False, out[1].data_ptr(), s.cuda_stream)
    s.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        ctx.intersect_device(n, dr.data_ptr(), 0.0, False, out[2].data_ptr(), s.cuda_stream)
    ctx.intersect_device(n, dr.data_ptr(), 0.0, False, out[0].data_ptr(), s.cuda_stream)
    g.replay()
    torch.cuda.synchronize()
    host = out.cpu().numpy()
    for k, label in enumerate(("list", "no allocation", "captured")):
        h = np.ascontiguousarray(host[k]).view(hr.HIT_DTYPE).reshape(-1)
        compare(h, ref, f"{label} {kinds} {modes}")
    assert (ref["kind"] > 0).any()
