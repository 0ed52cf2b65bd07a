"""What a program does with this renderer, as cases that can be timed.

A program loads or makes a mesh of curved hexahedra with a modal field, builds
the tree once, and then sends rays through it for as long as it runs: pictures
from moving cameras at changing isovalues, batches of rays of its own, many
views at once, paths with bounces. So a case keeps the context (scene, tree,
trained network) as such a program keeps it, and every seed brings another
camera, other rays and other isovalues. The scenes are this repository's own
workloads: grids of curved hexahedra over the unit cube (P = 4 on 4^3, P = 6
on 32^3, P = 2..8 mixed on 48^3, P = 5 on 64^3) and the sheet of prisms, quads
and triangles. They are made here, in 64 bits, and handed over through
ho_add_hexes, so that exact() can trace the same coefficients itself.

Of a hit every field comes back but `iters`, which counts the solver's steps
and is no answer; `flags` come back where they are the same in every run (with
network starts they say which start failed, which depends on the order in
which the solves of an element finish).
"""
from __future__ import annotations

import math
import os
import sys
from collections import OrderedDict
from functools import lru_cache

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "test-_gb300"))

import horender as hr  # noqa: E402
import prim_synth  # noqa: E402

DEV = "cuda"
# grid side, orders, curving amplitude over h, Gaussians in the field, isovalues
SCENES = {
    "hex4_p4": (4, 4, 4, 0.05, 8, [0.2]),
    "hex32_p6": (32, 6, 6, 0.08, 64, [-0.3, 0.0, 0.3]),
    "hex48_mixed": (48, 2, 8, 0.10, 64, [-0.2, 0.1, 0.3]),
    "hex64_p5": (64, 5, 5, 0.12, 64, [0.1]),
}


def listed():
    return [
        # a probe: a few hundred rays of the caller's own, where launches and latency are all there is
        dict(name="rays_probe", kind="rays", scene="hex4_p4", mode="batched", n=777),
        # the small picture of a first look at a mesh
        dict(name="image_small", kind="image", scene="hex4_p4", mode="batched", w=256, h=256, isos=1),
        # the allocation-free call of a program whose own pool holds the device's memory
        dict(name="rays_noalloc", kind="noalloc", scene="hex32_p6", mode="batched", n=20011),
        # incoherent rays (probing, light transport written elsewhere) through a fine mesh
        dict(name="rays_large", kind="rays", scene="hex32_p6", mode="batched", n=1000003),
        # the ordinary picture: full HD, three nested isosurfaces, cold starts (the default mode)
        dict(name="image_hd", kind="image", scene="hex32_p6", mode="batched", w=1920, h=1080, isos=3),
        # the same picture from a context with a trained network
        dict(name="image_hd_learned", kind="image", scene="hex32_p6", mode="learned", w=1920, h=1080, isos=3),
        # a mesh refined in p: every order from 2 to 8 in one picture
        dict(name="image_mixed", kind="image", scene="hex48_mixed", mode="batched", w=1024, h=1024, isos=3),
        # an animation's frames in one call, of different sizes, 1 to 3 isovalues each
        dict(name="views_mixed", kind="views", scene="hex48_mixed", mode="batched", views=12, top=1024),
        # the repository's headline scene and size: 4K, 64^3 elements
        dict(name="image_4k", kind="image", scene="hex64_p5", mode="batched", w=3840, h=2160, isos=1),
        # the reference's own render loop: diffuse bounces, one sample a pixel and pass
        dict(name="paths", kind="path", scene="hex32_p6", mode="batched", w=640, h=360, depth=4),
        # a scene of prisms, quads and curved triangles
        dict(name="prims_image", kind="prims", side=64, w=960, h=540),
        # the network's training step (forward, loss, every gradient)
        dict(name="net_grad", kind="grad", n=4096),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["rays", "image", "image", "noalloc", "views", "path", "prims", "grad"])
    if kind == "grad":
        return dict(kind="grad", n=log(64, 16384))
    if kind == "prims":
        return dict(kind="prims", side=rng.choice([8, 16, 32, 64]), w=log(48, 960), h=log(33, 540))
    if kind == "views":
        return dict(kind="views", scene="hex48_mixed", mode="batched", views=rng.randint(2, 12), top=log(64, 1024))
    if kind == "path":
        return dict(kind="path", scene=rng.choice(["hex4_p4", "hex32_p6"]), mode="batched", w=log(40, 640),
                    h=log(30, 360), depth=rng.randint(1, 4))
    scene = rng.choice(["hex4_p4", "hex32_p6", "hex48_mixed"])
    if kind == "noalloc":
        return dict(kind="noalloc", scene=scene, mode="batched", n=log(1, 32768))
    if kind == "rays":
        return dict(kind="rays", scene=scene, mode="batched", n=log(1, 1000003))
    mode = "batched" if scene == "hex48_mixed" else rng.choice(["batched", "learned"])
    return dict(kind="image", scene=scene, mode=mode, w=log(33, 1920), h=log(17, 1080), isos=rng.randint(1, 3))


# ---------------------------------------------------------------------------
# Scenes: coefficients in the Modified-A basis, fitted in 64 bits at GLL nodes
# ---------------------------------------------------------------------------
def basis(x, n):
    """Modified-A modes 0..n-1 and their derivatives at x, stacked last."""
    one = torch.ones_like(x)
    v, d = [0.5 * (1 - x), 0.5 * (1 + x)], [-0.5 * one, 0.5 * one]
    w, dw = 0.25 * (1 - x * x), -0.5 * x
    p0, p1, q0, q1 = one, 2 * x, 0 * one, 2 * one
    for m in range(n - 2):
        v.append(w * p0)
        d.append(dw * p0 + w * q0)
        a, b = (2 * m + 5) * (m + 3) / ((m + 2) * (m + 4)), (m + 3) / (m + 4)
        p0, p1, q0, q1 = p1, a * x * p1 - b * p0, q1, a * (p1 + x * q1) - b * q0
    return torch.stack(v[:n], -1), torch.stack(d[:n], -1)


@lru_cache(maxsize=None)
def gll(n):
    """GLL nodes on [-1, 1] and the inverse of the modal Vandermonde matrix."""
    c = np.zeros(n)
    c[-1] = 1
    x = np.concatenate([[-1.0], np.sort(np.polynomial.legendre.legroots(np.polynomial.legendre.legder(c)).real), [1.0]])
    inv = np.linalg.inv(basis(torch.from_numpy(x), n)[0].numpy())
    return x, inv


@lru_cache(maxsize=1)
def scene_arrays(name):
    """ho_add_hexes' arguments for one of SCENES (numpy, FP32 coefficients)."""
    side, p_min, p_max, amp, n_gauss, _ = SCENES[name]
    g = np.random.default_rng(20 + side)
    cen = torch.from_numpy(g.uniform(0, 1, (n_gauss, 3))).to(DEV)
    wid = torch.from_numpy(0.5 / g.uniform(0.1, 0.3, n_gauss) ** 2).to(DEV)
    height = torch.from_numpy(g.uniform(-1, 1, n_gauss)).to(DEV)
    ne, h = side ** 3, 1.0 / side
    order = g.integers(p_min, p_max + 1, ne) + 1
    size = order.astype(np.int64) ** 3
    field_off = np.concatenate([[0], np.cumsum(size)[:-1]])
    geom, field = np.zeros(3 * int(size.sum()), np.float32), np.zeros(int(size.sum()), np.float32)

    def place(q):  # the curved mesh: q + amp h sin sin sin, the same shift in x, y and z
        return q + amp * h * torch.sin(2 * math.pi * q).prod(-1, keepdim=True)

    def cell(e):
        e = torch.from_numpy(e).to(DEV)
        return torch.stack([e % side, (e // side) % side, e // (side * side)], -1).double()

    for n in np.unique(order):
        x, inv = gll(int(n))
        x, inv = torch.from_numpy(x).to(DEV), torch.from_numpy(inv).to(DEV)
        node = torch.stack(torch.meshgrid(x, x, x, indexing="ij")[::-1], -1).reshape(-1, 3)  # (k, j, i), x fastest
        of = np.nonzero(order == n)[0]
        for at in np.array_split(of, max(1, len(of) * int(n) ** 3 // 4_000_000)):
            p = place((cell(at)[:, None] + 0.5 * (node + 1)) * h)
            u = torch.zeros(p.shape[:2], dtype=torch.float64, device=DEV)
            for c, w, a in zip(cen, wid, height):
                u += a * torch.exp(-w * (p - c).square().sum(-1))
            val = torch.cat([p, u[..., None]], -1).permute(0, 2, 1).reshape(len(at), 4, n, n, n)
            co = torch.einsum("ecKJI,kK,jJ,iI->eckji", val, inv, inv, inv).float().cpu().numpy().reshape(len(at), 4, -1)
            s = int(n) ** 3
            geom[(3 * field_off[at])[:, None] + np.arange(3 * s)] = co[:, :3].reshape(len(at), -1)
            field[field_off[at][:, None] + np.arange(s)] = co[:, 3]
    xml = torch.tensor([(0, 0, 0), (1, 0, 0), (1, 1, 0), (0, 1, 0), (0, 0, 1), (1, 0, 1), (1, 1, 1), (0, 1, 1)],
                       dtype=torch.float64, device=DEV)
    corners = place((cell(np.arange(ne))[:, None] + xml) * h).float().cpu().numpy()
    modes = np.repeat(order.astype(np.uint32)[:, None], 3, 1)
    return dict(corners=corners, geom_modes=modes, geom=geom, geom_offsets=3 * field_off, field_modes=modes, field=field,
                field_offsets=field_off)


def train(ctx):
    """A network for the context's scene from its own training pairs, the same
    in every run (the library's trainer adds in any order, so its networks
    differ from run to run in the last bits)."""
    X, T, V = (torch.from_numpy(a).to(DEV) for a in ctx.learn_samples(400_000, 3))
    X, T = X[V > 0], T[V > 0][:, :6]
    g = torch.Generator(device="cpu").manual_seed(5)
    dims = [(48, 128), (128, 128), (128, 128), (128, 8)]
    par = []
    for i, o in dims:
        par += [(torch.randn(i, o, generator=g) * math.sqrt(2.0 / i)).to(DEV), torch.zeros(o, device=DEV)]
    for p in par:
        p.requires_grad_(True)
    opt = torch.optim.Adam(par, lr=2e-3)
    steps = 800
    rows = torch.randint(0, X.shape[0], (steps, 4096), generator=g).to(DEV)
    for k in range(steps):
        for group in opt.param_groups:
            group["lr"] = 2e-3 * (0.05 + 0.475 * (1 + math.cos(math.pi * k / steps)))
        y = X[rows[k]]
        for layer in range(4):
            y = y @ par[2 * layer] + par[2 * layer + 1]
            y = torch.nn.functional.gelu(y, approximate="tanh") if layer < 3 else y
        opt.zero_grad()
        (y[:, :6] - T[rows[k]]).square().sum(1).mean().backward()
        opt.step()
    ctx.mlp_set_params(torch.cat([p.detach().reshape(-1) for p in par]).cpu().numpy())


_CONTEXTS: OrderedDict = OrderedDict()


def context(scene, mode):
    """The context of a running program: the last scene's is kept."""
    if (scene, mode) not in _CONTEXTS:
        _CONTEXTS.clear()
        ctx = hr.Context(0)
        if scene.startswith("prims"):
            ctx.add_prim_arrays(prim_synth.mixed_scene(seed=11, n_side=int(scene[5:])))
        else:
            ctx.add_hexes(**scene_arrays(scene))
        ctx.build_bvh()
        if mode == "learned":
            train(ctx)
        ctx.set_mode({"batched": hr.MODE_BATCHED, "learned": hr.MODE_LEARNED}[mode])
        _CONTEXTS[scene, mode] = ctx
    return _CONTEXTS[scene, mode]


# ---------------------------------------------------------------------------
# A case's inputs
# ---------------------------------------------------------------------------
def camera(rng):
    """A camera on a sphere around the cube, looking near its centre."""
    y, phi, r = rng.uniform(-0.7, 0.7), rng.uniform(0, 2 * math.pi), rng.uniform(2.1, 3.2)
    c = math.sqrt(1 - y * y)
    at = 0.5 + rng.uniform(-0.1, 0.1, 3)
    pos = at + r * np.array([c * math.cos(phi), y, c * math.sin(phi)])
    return hr.Camera(tuple(float(v) for v in pos), tuple(float(v) for v in at), (0, 1, 0), float(rng.uniform(35, 60)))


def isovalues(scene, n, rng):
    return [float(np.float32(v + rng.uniform(-0.05, 0.05))) for v in SCENES[scene][5][:n]] + [
        float(np.float32(rng.uniform(-0.4, 0.4))) for _ in range(n - len(SCENES[scene][5]))]


def rays_of(n, rng):
    """Rays from a sphere around the cube to points within it."""
    o = rng.normal(size=(n, 3))
    o = 0.5 + 1.5 * o / np.linalg.norm(o, axis=1, keepdims=True)
    d = rng.uniform(0, 1, (n, 3)) - o
    return np.concatenate([o, d / np.linalg.norm(d, axis=1, keepdims=True)], 1).astype(np.float32)


def buffers(n, rgb):
    return dict(hits=torch.zeros((n, 12), dtype=torch.int32, device=DEV),
                rgb=torch.zeros((n, 3), dtype=torch.uint8, device=DEV) if rgb else None)


def view_sizes(case):
    """Widths, heights and numbers of isovalues of a call's views."""
    top, k = case["top"], range(case["views"])
    return [(top // 4, top // 2, 5 * top // 8, top)[i % 4] for i in k], [
        (top // 4, top // 2, 11 * top // 31, top)[i % 4] for i in k], [1 + i % 3 for i in k]


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    if kind == "grad":
        ctx = hr.Context(0)
        ctx.mlp_init(int(rng.integers(1 << 30)))
        n = case["n"]
        return dict(case=case, ctx=ctx, X=rng.normal(size=(n, 48)).astype(np.float32),
                    T=rng.normal(size=(n, 8)).astype(np.float32), V=(rng.uniform(size=n) > 0.1).astype(np.uint8))
    if kind == "prims":
        ctx = context("prims%d" % case["side"], "batched")
        cam = hr.Camera((1.6 + float(rng.uniform(-0.3, 0.3)), 1.1 + float(rng.uniform(-0.2, 0.4)),
                         1.9 + float(rng.uniform(-0.3, 0.3))), (0.5, 0.2, 0.3), (0, 1, 0), 50.0)
        return dict(case=case, ctx=ctx, cam=cam, **buffers(case["w"] * case["h"], True))
    ctx = context(case["scene"], case["mode"])
    s = dict(case=case, ctx=ctx)
    if kind in ("rays", "noalloc"):
        s["rays"] = torch.from_numpy(rays_of(case["n"], rng)).to(DEV)
        s["isos"] = isovalues(case["scene"], 1, rng)
        s.update(buffers(case["n"], False))
    elif kind == "image":
        s["cam"], s["isos"] = camera(rng), isovalues(case["scene"], case["isos"], rng)
        s.update(buffers(case["w"] * case["h"] * case["isos"], True))
    elif kind == "path":
        s["cam"], s["isos"] = camera(rng), isovalues(case["scene"], 1, rng)
        s["path_seed"] = int(rng.integers(1 << 30))
        s["rgb"] = torch.zeros((case["h"], case["w"], 3), dtype=torch.uint8, device=DEV)
    elif kind == "views":
        s["w"], s["h"], n = view_sizes(case)
        s["cams"] = [camera(rng) for _ in n]
        s["isos"] = [isovalues(case["scene"], k, rng) for k in n]
        s.update(buffers(sum(w * h * len(i) for w, h, i in zip(s["w"], s["h"], s["isos"])), True))
    return s


def hit_fields(s, flags):
    """ho_hit's fields as views of the caller's buffer of hits."""
    i, f = s["hits"], s["hits"].view(torch.float32)
    out = dict(t=f[:, 0], elem=i[:, 1], face_kind=i.view(torch.int16)[:, 4:6], xi=f[:, 3:6], n=f[:, 6:9], u=f[:, 9])
    if flags:
        out["flags"] = i[:, 10]
    if s.get("rgb") is not None:
        out["rgb"] = s["rgb"]
    return out


def run(s):
    case, ctx = s["case"], s["ctx"]
    kind = case["kind"]
    if kind == "grad":
        loss, grads = ctx.mlp_grad(s["X"], s["T"], s["V"])
        return dict(loss=loss, grads=grads)
    stream = torch.cuda.current_stream().cuda_stream or None
    if kind == "path":
        n = ctx.path_trace_device(s["cam"], s["isos"], case["w"], case["h"], s["rgb"].data_ptr(), stream, spp=1,
                                  max_depth=case["depth"], seed=s["path_seed"], iso_zero_disables=False)
        return dict(rgb=s["rgb"], rays=n)
    hits = s["hits"].data_ptr()
    if kind == "rays":
        ctx.intersect_device(case["n"], s["rays"].data_ptr(), s["isos"][0], True, hits, stream)
    elif kind == "noalloc":
        ctx.intersect_device_noalloc(case["n"], s["rays"].data_ptr(), s["isos"][0], True, hits, stream)
    elif kind == "views":
        ctx.render_views_device(s["cams"], s["w"], s["h"], s["isos"], s["rgb"].data_ptr(), hits, stream)
    elif kind == "prims":
        ctx.render_device(s["cam"], [0.0], case["w"], case["h"], s["rgb"].data_ptr(), hits, stream)
    else:
        ctx.render_device(s["cam"], s["isos"], case["w"], case["h"], s["rgb"].data_ptr(), hits, stream,
                          iso_zero_disables=False)
    return hit_fields(s, case.get("mode") != "learned")


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    """Bytes: the outputs, caller's rays and the scene's records, once each.
    FLOPs: for the share of the rays that meets the cube (a third of a
    picture, all of the caller's rays), one point and Jacobian evaluation for
    each of three Newton steps and the check of the hit; for primitives, the
    same at 27 coefficients; for the network its products, forward and back."""
    kind = case["kind"]
    if kind == "grad":
        macs = 48 * 128 + 2 * 128 * 128 + 128 * 8
        return dict(bytes=case["n"] * (48 + 8) * 4 + 2 * 4 * macs, flops=6 * macs * case["n"])
    if kind == "prims":
        q = case["w"] * case["h"]
        return dict(bytes=q * 51 + 3.5 * case["side"] ** 2 * (128 + 160), flops=q * 4 * 3 * 27 * 8)
    side, p_min, p_max = SCENES[case["scene"]][:3]
    n3 = np.mean([(p + 1) ** 3 for p in range(p_min, p_max + 1)])
    if kind in ("rays", "noalloc"):
        q, out = case["n"], 24 + 48
        met = q
    elif kind == "image":
        q, out = case["w"] * case["h"] * case["isos"], 51
        met = q / 3
    elif kind == "path":
        q, out = case["w"] * case["h"], 3
        met = q / 3 * case["depth"]
    else:
        q, out = sum(w * h * n for w, h, n in zip(*view_sizes(case))), 51
        met = q / 3
    return dict(bytes=q * out + min(side ** 3, met) * 16 * n3, flops=met * 4 * 3 * 4 * n3)


# ---------------------------------------------------------------------------
# The same answers in 64 bits
# ---------------------------------------------------------------------------
def bf16(x):
    """Rounded to BF16, as the network keeps its operands."""
    return x.to(torch.bfloat16).double()


def exact_grad(case, seed):
    s = prepare(case, seed)
    flat = torch.from_numpy(s["ctx"].mlp_params()).to(DEV)
    X, T, V = (torch.from_numpy(s[k]).to(DEV) for k in "XTV")
    par, at = [], 0
    for i, o in [(48, 128), (128, 128), (128, 128), (128, 8)]:
        par.append((bf16(flat[at:at + i * o].reshape(i, o)), flat[at + i * o:at + i * o + o].double()))
        at += i * o + o
    hs, zs = [bf16(X)], []
    for layer, (W, b) in enumerate(par):
        zs.append((hs[-1] @ W + b).requires_grad_(True))
        if layer < 3:
            hs.append(bf16(torch.nn.functional.gelu(zs[-1], approximate="tanh").detach()))
    d = (zs[-1] - T.double()).detach()
    d[:, 6:] = 0
    d[V == 0] = 0
    n = max(1, int(V.sum()))
    dz, grads = 2 * d / n, [None] * 4
    for layer in (3, 2, 1, 0):
        grads[layer] = torch.cat([(hs[layer].T @ bf16(dz)).reshape(-1), dz.sum(0)])
        if layer:
            dh, z = bf16(dz) @ par[layer][0].T, zs[layer - 1]
            dz = dh * torch.autograd.grad(torch.nn.functional.gelu(z, approximate="tanh").sum(), z)[0]
    return dict(loss=float((d * d).sum() / n), grads=torch.cat(grads).cpu().numpy())


class Elements:
    """The scene's coefficients in 64 bits (one order): x, y, z and the field."""

    def __init__(self, name):
        a = scene_arrays(name)
        n = self.n = int(a["geom_modes"][0, 0])
        ne = len(a["geom_offsets"])
        g = torch.from_numpy(a["geom"]).reshape(ne, 3, n, n, n)
        self.c = torch.cat([g, torch.from_numpy(a["field"]).reshape(ne, 1, n, n, n)], 1).to(DEV).double()
        x = torch.linspace(-1, 1, max(4, n + 2), dtype=torch.float64, device=DEV)
        b = basis(x, n)[0]
        p = torch.einsum("eckji,Kk,Jj,Ii->ecKJI", self.c[:, :3], b, b, b).reshape(ne, 3, -1)
        lo, hi = p.amin(-1), p.amax(-1)
        pad = ((hi - lo) * 0.15).clamp(min=1e-3)  # the candidates' boxes: the sampled box and 15% on each side
        self.lo, self.hi = lo - pad, hi + pad

    def at(self, e, xi):
        """x, y, z, u and their three partials at xi of elements e: (m, 4, 4)."""
        out = []
        for k in range(0, len(e), 400_000):
            c = self.c[e[k:k + 400_000]]
            (a, da), (b, db), (g, dg) = (basis(xi[k:k + 400_000, q], self.n) for q in range(3))
            i = torch.stack([a, da], -1)
            s = (c.reshape(len(c), -1, self.n) @ i).reshape(len(c), 4, self.n, self.n, 2)
            j = torch.einsum("mckjd,mj->mckd", s, b), torch.einsum("mckj,mj->mck", s[..., 0], db)
            out.append(torch.stack([torch.einsum("mck,mk->mc", j[0][..., 0], g), torch.einsum("mck,mk->mc", j[0][..., 1], g),
                                    torch.einsum("mck,mk->mc", j[1], g), torch.einsum("mck,mk->mc", j[0][..., 0], dg)], -1))
        return torch.cat(out) if out else torch.zeros((0, 4, 4), dtype=torch.float64, device=DEV)


def newton(el, e, target, xi, steps=50):
    """The inverse map by Newton's method: xi, and where it converged."""
    ok = torch.zeros(len(e), dtype=torch.bool, device=DEV)
    for _ in range(steps):
        live = torch.nonzero(~ok & xi.isfinite().all(-1))[:, 0]
        if not len(live):
            break
        v = el.at(e[live], xi[live])
        dx = torch.linalg.solve_ex(v[:, :3, 1:], (v[:, :3, 0] - target[live])[..., None])[0][..., 0]
        xi = xi.index_put((live,), xi[live] - dx)
        ok = ok.index_put((live,), dx.abs().amax(-1) < 1e-5)
    return xi, ok


def field_along(el, e, o, d, t, xi, iso):
    """u - iso at the point t of each ray, its slope in t, xi, the gradient."""
    xi, ok = newton(el, e, o + t[:, None] * d, xi)
    v = el.at(e, xi)
    grad = torch.linalg.solve_ex(v[:, :3, 1:].transpose(1, 2), v[:, 3, 1:, None])[0][..., 0]
    return v[:, 3, 0] - iso, (grad * d).sum(-1), xi, grad, ok


FACES = [(2, -1.0, 0, 1), (1, -1.0, 0, 2), (0, 1.0, 1, 2), (1, 1.0, 0, 2), (0, -1.0, 1, 2), (2, 1.0, 0, 1)]


def iso_hit(el, e, o, d, te, tx, iso):
    """First sign change over 17 samples of the segment, then its root."""
    m, k = len(e), torch.arange(17, dtype=torch.float64, device=DEV) / 16
    t = te[:, None] + (tx - te)[:, None] * k
    rep = torch.arange(m, device=DEV).repeat_interleave(17)
    f, _, xi, _, ok = field_along(el, e[rep], o[rep], d[rep], t.reshape(-1), torch.zeros((17 * m, 3), dtype=torch.float64,
                                                                                     device=DEV), iso)
    f, ok, xi = f.reshape(m, 17), ok.reshape(m, 17), xi.reshape(m, 17, 3)
    prev = torch.full((m,), -1, device=DEV)
    left, right = prev.clone(), prev.clone()
    row = torch.arange(m, device=DEV)
    for i in range(17):
        change = ok[:, i] & (prev >= 0) & (right < 0) & (f[row, prev.clamp(min=0)] * f[:, i] <= 0)
        left, right = torch.where(change, prev, left), torch.where(change, i, right)
        prev = torch.where(ok[:, i], i, prev)
    at = torch.nonzero(right >= 0)[:, 0]
    lo, hi, fl = t[at, left[at]], t[at, right[at]], f[at, left[at]]
    x, root, g = xi[at, left[at]], 0.5 * (lo + hi), torch.zeros((len(at), 3), dtype=torch.float64, device=DEV)
    for _ in range(60):  # bisection with Newton steps where they stay inside
        fm, slope, x, g, _ = field_along(el, e[at], o[at], d[at], root, x, iso)
        same = fl * fm > 0
        lo, hi = torch.where(same, root, lo), torch.where(same, hi, root)
        step = root - fm / slope
        root = torch.where((step > lo) & (step < hi), step, torch.where(fm.abs() < 1e-13, root, 0.5 * (lo + hi)))
    return at, root, x, g


def face_hit(el, e, o, d, best):
    """Nearest of the six faces: the first of nine starts that converges."""
    m = len(e)
    t = torch.full((m,), math.inf, dtype=torch.float64, device=DEV)
    face, xi = torch.full((m,), -1, device=DEV), torch.zeros((m, 3), dtype=torch.float64, device=DEV)

    def step(q, p, tau, f):
        fixed, _, a, b = FACES[f]
        v = el.at(e[q], p)[:, :3]
        r = v[..., 0] - (o[q] + tau[:, None] * d[q])
        M = torch.stack([v[..., 1 + a], v[..., 1 + b], -d[q]], -1)
        return r.abs().amax(-1), -torch.linalg.solve_ex(M, r[..., None])[0][..., 0]

    for f, (fixed, side, a, b) in enumerate(FACES):
        todo = torch.arange(m, device=DEV)
        for s in range(9):
            p = torch.zeros((len(todo), 3), dtype=torch.float64, device=DEV)
            p[:, fixed], p[:, a], p[:, b] = side, (-0.8, 0.0, 0.8)[s % 3], (-0.8, 0.0, 0.8)[s // 3]
            tau = ((el.at(e[todo], p)[:, :3, 0] - o[todo]) * d[todo]).sum(-1) / d[todo].square().sum(-1)
            tau = torch.minimum(tau.clamp(min=1e-3), best[todo])
            live, got = torch.arange(len(todo), device=DEV), torch.zeros(len(todo), dtype=torch.bool, device=DEV)
            last = torch.full((len(todo),), math.inf, dtype=torch.float64, device=DEV)
            for it in range(50):
                if not len(live):
                    break
                r, dx = step(todo[live], p[live], tau[live], f)
                near = r < 1e-4
                got[live[near & (p[live][:, a].abs() <= 1.001) & (p[live][:, b].abs() <= 1.001)]] = True
                on = ~near & ~((r > 1.5 * last[live]) if it > 5 else near)
                last[live] = r
                live, dx = live[on], dx[on]
                dx = dx * (0.25 / dx.abs().amax(-1, keepdim=True)).clamp(max=1.0)
                tau[live] = torch.minimum((tau[live] + dx[:, 2]).clamp(min=1e-3), best[todo[live]])
                p[live, a] = (p[live, a] + dx[:, 0]).clamp(-1.5, 1.5)
                p[live, b] = (p[live, b] + dx[:, 1]).clamp(-1.5, 1.5)
            for _ in range(4):  # to the root itself
                _, dx = step(todo[got], p[got], tau[got], f)
                p[got, a], p[got, b], tau[got] = p[got, a] + dx[:, 0], p[got, b] + dx[:, 1], tau[got] + dx[:, 2]
            q = todo[got]
            nearer = tau[got] < torch.minimum(t[q], best[q])
            t[q[nearer]], face[q[nearer]], xi[q[nearer]] = tau[got][nearer], f, p[got][nearer]
            todo = todo[~got]
    return t, face, xi


def exact_hits(el, rays, iso):
    """Every ray's answer: its candidate elements in the order of their boxes'
    entries, in each the isosurface, else the nearest face."""
    o, d = rays[:, :3], rays[:, 3:]
    ta, tb = (el.lo[None] - o[:, None]) / d[:, None], (el.hi[None] - o[:, None]) / d[:, None]
    enter, leave = torch.minimum(ta, tb).amax(-1).clamp(min=1e-3), torch.maximum(ta, tb).amin(-1)
    enter = torch.where(leave >= enter, enter, math.inf)
    key, of = enter.sort(dim=1, stable=True)
    n = len(rays)
    best = torch.full((n,), float(np.finfo(np.float32).max), dtype=torch.float64, device=DEV)
    xi, nrm = torch.zeros((2, n, 3), dtype=torch.float64, device=DEV)
    u = torch.zeros(n, dtype=torch.float64, device=DEV)

    def keep(r, t, x, g, val):
        g = g / g.norm(dim=-1, keepdim=True)
        g = torch.where(((g * d[r]).sum(-1) > 0)[:, None], -g, g)
        best[r], xi[r], nrm[r], u[r] = t, x, g, val

    for k in range(key.shape[1]):
        r = torch.nonzero(key[:, k] < best)[:, 0]
        r = r[key[r, k].isfinite()]
        if not len(r):
            break
        e = of[r, k]
        at, t, x, g = iso_hit(el, e, o[r], d[r], key[r, k], torch.minimum(leave[r, e], best[r]), iso)
        none = torch.ones(len(r), dtype=torch.bool, device=DEV)
        none[at] = False
        new = t < best[r[at]]
        keep(r[at][new], t[new], x[new], g[new], torch.full((int(new.sum()),), iso, dtype=torch.float64, device=DEV))
        r, e = r[none], e[none]
        t, face, x = face_hit(el, e, o[r], d[r], best[r])
        hit = face >= 0
        r, e, t, x = r[hit], e[hit], t[hit], x[hit]
        v = el.at(e, x)
        dr, ds, dt = v[:, :3, 1], v[:, :3, 2], v[:, :3, 3]
        g = torch.where((x[:, :1].abs() > 0.9), torch.linalg.cross(ds, dt),
                        torch.where((x[:, 1:2].abs() > 0.9), torch.linalg.cross(dr, dt), torch.linalg.cross(dr, ds)))
        keep(r, t, x, g, v[:, 3, 0])
    return dict(t=best, xi=xi, n=nrm, u=u)


def camera_rays(cam, w, h):
    """Pixel-centre rays of a pinhole camera, from the FP32 values a caller gives."""
    f = np.float32
    pos, at, up = (np.array(v, f).astype(np.float64) for v in (cam.lookfrom, cam.lookat, cam.vup))
    back = pos - at
    focus = np.linalg.norm(back)
    back = back / focus
    right = np.cross(up, back)
    right /= np.linalg.norm(right)
    high = 2 * math.tan(math.radians(float(f(cam.vfov_deg))) / 2)
    x, y = np.meshgrid((np.arange(w) + 0.5) / w - 0.5, (np.arange(h) + 0.5) / h - 0.5)
    d = x[..., None] * right * high * w / h + y[..., None] * np.cross(back, right) * high - back
    d = (d / np.linalg.norm(d, axis=-1, keepdims=True)).reshape(-1, 3)
    return np.concatenate([np.broadcast_to(pos, d.shape), d], 1)


def exact(case, seed):
    """Of the network's gradients, and of rays and small pictures through the
    coarse mesh; tracing the fine meshes in 64 bits takes minutes, and the
    other kinds (paths and the primitives' start searches, which branch on
    32-bit values) have no value in 64 bits."""
    if case["kind"] == "grad":
        return exact_grad(case, seed)
    if case.get("scene") != "hex4_p4" or case["kind"] not in ("rays", "image"):
        return None
    rng = np.random.default_rng(seed)
    if case["kind"] == "rays":
        if case["n"] > 70_000:
            return None
        rays, isos = rays_of(case["n"], rng).astype(np.float64), isovalues(case["scene"], 1, rng)
    else:
        if case["w"] * case["h"] * case["isos"] > 70_000:
            return None
        cam = camera(rng)
        rays, isos = camera_rays(cam, case["w"], case["h"]), isovalues(case["scene"], case["isos"], rng)
    el = Elements(case["scene"])
    r = torch.from_numpy(rays).to(DEV)
    got = [exact_hits(el, r, v) for v in isos]
    # where two elements share the surface point, rounding says which one is
    # named, and xi is in the one that is: no value in 64 bits
    out = {k: torch.cat([g[k] for g in got]).cpu().numpy() for k in ("t", "n", "u")}
    out.update(xi=None, elem=None, face_kind=None, flags=None, rgb=None)
    return out
