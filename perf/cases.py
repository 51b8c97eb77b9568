"""The measured cases: the pipeline's stages as a user's program calls them.

A capture goes through Stage 1 (cubes of each depth map), Stage 2 (merge),
Stage 3 (2:1 balance), Stage 5 (histograms), the learned warm start, Stage 6
(the TGV solve) and Stage 7 (surface).  Each case is one call of one stage on
seeded synthetic input of the shapes that the package's configurations
(`tgvreconclaude_gb300/workloads.py`) and tests use: the torus16 shape (16
maps of 640x480, depth <= 8, 300 iterations), the three64 shape (64 maps of
1920x1080, depth <= 11, 1000 iterations) and the chunked terrain shape (64
chunks, solved to a relative residual of 1e-4), with the small octrees of the
tests below them.

listed(), draw(rng), prepare(case, seed), run(state), work(case) and
exact(case, seed).
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from tgvreconclaude_gb300 import _native as N, api, formats as F, scenes as S, workloads as W
from tgvreconclaude_gb300 import warmstart as WS

DEV = "cuda"
# the scenes' surface areas and half box sides
AREA = dict(torus=11.8, three=26.5, terrain=62.0, balls=16.9)
ROOT = dict(torus=1.5, three=3.0, terrain=4.0, balls=2.0)


def listed():
    return [
        # the smallest solve: a test-sized octree through the reference's own entry point, default
        # parameters; latency and launches are all of it
        dict(name="solve_tiny", kind="solve", where="host", mode="inmem", scene="octree", cubes=1200, depth=5,
             nbins=8, iters=200, alpha0=0.02, alpha1=0.04, tol=0.0),
        # one object in one chunk, the torus16 shape, inputs and result on the device
        dict(name="solve_object", kind="solve", where="device", mode="inmem", scene="torus", cubes=266_000,
             samples=1_500_000, depth=8, nbins=10, iters=300, alpha0=2.0, alpha1=1.0, tol=0.0),
        # a whole multi-object capture, the three64 shape: the largest solve
        dict(name="solve_capture", kind="solve", where="device", mode="inmem", scene="three", cubes=6_000_000,
             samples=14_000_000, depth=11, nbins=10, iters=1000, alpha0=2.0, alpha1=1.0, tol=0.0),
        # out-of-core semantics: 64 chunks of a terrain solved to a tolerance, all chunks of a level together
        dict(name="solve_chunks", kind="solve", where="device", mode="stream", scene="terrain", cubes=2_800_000,
             samples=6_000_000, depth=10, nbins=10, iters=6000, alpha0=2.0, alpha1=1.0, tol=1e-4, chunks=64),
        # histograms of one object's cubes from its maps, host arrays in and out (the torus16 shape)
        dict(name="hist_object", kind="hist_host", maps=16, width=640, height=480, cubes=150_000, samples=1_500_000,
             depth=8, nbins=10),
        # histograms of a capture, pyramids and cubes resident on the device (64 maps of 1920x1080)
        dict(name="hist_capture", kind="hist_dev", maps=64, width=1920, height=1080, cubes=2_000_000,
             samples=8_000_000, depth=10, nbins=10),
        # Stage 1: the cubes of one full-size depth map
        dict(name="cubes_of_map", kind="stage1", width=1920, height=1080, sigma=0.004),
        # Stage 2: the sorted cube lists of 16 maps merged into one
        dict(name="merge_maps", kind="merge", lists=16, per_list=400_000, depth=10),
        # Stage 3: 2:1 balance of a merged list
        dict(name="balance_capture", kind="balance", scene="three", cubes=1_200_000, samples=3_000_000, depth=10),
        # Stage 7: the iso-surface of a solved octree with vertex normals, host arrays in and out
        dict(name="surface_capture", kind="surface", scene="three", cubes=1_900_000, samples=6_000_000, depth=10),
        # the learned warm start's prediction for every cube of a chunked capture
        dict(name="warm_start", kind="mlp_infer", scene="three", cubes=2_200_000, samples=8_000_000, depth=10,
             nbins=10, chunks=128),
        # its training direction: the gradient of the loss over a data set of feature rows
        dict(name="warm_start_gradient", kind="mlp_grad", rows=400_000, nbins=10),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _size(rng, scene, lo, hi):
    """Cubes, samples and depth of a generated octree: a depth at which the
    samples make more cubes than are taken."""
    n = _log(rng, lo, hi)
    samples = int(n / 0.3)
    d = 6
    while 6 * AREA[scene] / (2 * ROOT[scene] / (1 << d)) ** 2 < samples and d < 11:
        d += 1
    return dict(cubes=n, samples=samples, depth=min(11, d + rng.randint(0, 1)))


def draw(rng):
    kind = rng.choice(["solve", "solve", "solve", "hist_host", "hist_dev", "stage1", "merge", "balance", "surface",
                       "mlp_infer", "mlp_grad"])
    nbins = rng.choice([8, 10])
    scene = rng.choice(["torus", "three", "terrain"])
    if kind == "solve":
        a = rng.choice([(0.02, 0.04), (2.0, 1.0)])
        c = dict(kind=kind, where=rng.choice(["host", "device"]), mode=rng.choice(["inmem", "inmem", "stream"]),
                 nbins=nbins, iters=rng.choice([rng.randint(50, 400), rng.randint(200, 1000)]), alpha0=a[0],
                 alpha1=a[1], tol=rng.choice([0.0, 0.0, 1e-4]))
        if rng.random() < 0.7:
            c |= dict(scene=scene) | _size(rng, scene, 6_000, 2_000_000)
        else:
            c |= dict(scene="octree", depth=5, cubes=_log(rng, 150, 2_000))
        if c["mode"] == "stream":
            c["chunks"] = _log(rng, 2, 64)
        return c
    if kind in ("hist_host", "hist_dev"):
        host = kind == "hist_host"
        w = _log(rng, 160, 1280 if host else 1920)
        return dict(kind=kind, maps=_log(rng, 2, 16 if host else 64), width=w,
                    height=max(31, int(w * rng.uniform(0.5, 0.56))), nbins=nbins) | _size(
                        rng, "balls", 6_000, 300_000 if host else 1_500_000)
    if kind == "stage1":
        w = _log(rng, 97, 1920)
        return dict(kind=kind, width=w, height=max(31, int(w * rng.uniform(0.45, 0.56))), sigma=rng.uniform(0.0, 0.01))
    if kind == "merge":
        k = _log(rng, 2, 64)
        return dict(kind=kind, lists=k, per_list=_log(rng, 1000, 6_000_000 // k), depth=rng.randint(7, 11))
    if kind == "mlp_grad":
        return dict(kind=kind, rows=_log(rng, 1000, 400_000), nbins=nbins)
    c = dict(kind=kind, scene=scene) | _size(rng, scene, 6_000, 1_000_000)
    if kind == "mlp_infer":
        c |= dict(nbins=nbins, chunks=_log(rng, 1, 128))
    return c


# --------------------------------------------------------------------- inputs ---

def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed))


def _objects(scene, seed):
    rng = np.random.default_rng(seed)
    if scene == "torus":
        return S.torus_scene(), (-1.5, -1.5, -1.5), 1.5
    if scene == "three":
        return S.three_objects_scene(rng), (-3.0, -3.0, -3.0), 3.0
    return S.terrain_scene(rng), (-4.0, -4.0, -4.0), 4.0


def _points(scene, n, seed):
    """n points on the scene's surfaces, uniform by area (terrain: by ground area)."""
    g = _gen(seed)
    prims, origin, r_root = _objects(scene, seed)
    area = {"sphere": lambda p: 4 * math.pi * p["r"] ** 2, "box": lambda p: 24 * p["h"] ** 2,
            "torus": lambda p: 4 * math.pi ** 2 * p["R"] * p["r"], "terrain": lambda p: 64.0}
    a = [area[p["kind"]](p) for p in prims]
    out = []
    for k, p in enumerate(prims):
        m = n - sum(len(o) for o in out) if k == len(prims) - 1 else int(n * a[k] / sum(a))
        u = torch.rand((m, 3), generator=g, device=DEV)
        if p["kind"] == "terrain":
            x, y = (u[:, 0] * 2 - 1) * 3.95, (u[:, 1] * 2 - 1) * 3.95
            z = torch.zeros_like(x)
            for A, kk, ph in zip(p["A"], p["k"], p["phi"]):
                z = z + A * torch.sin(kk[0] * x + kk[1] * y + ph)
            P = torch.stack([x, y, z], 1)
        elif p["kind"] == "sphere":
            d = torch.randn((m, 3), generator=g, device=DEV)
            P = p["r"] * d / d.norm(dim=1, keepdim=True)
        elif p["kind"] == "torus":
            t, s = 2 * math.pi * u[:, 0], 2 * math.pi * u[:, 1]
            q = p["R"] + p["r"] * torch.cos(s)
            P = torch.stack([q * torch.cos(t), q * torch.sin(t), p["r"] * torch.sin(s)], 1)
        else:  # box
            P = (u * 2 - 1) * p["h"]
            f = torch.randint(0, 6, (m,), generator=g, device=DEV)
            P[torch.arange(m, device=DEV), f % 3] = torch.where(f < 3, p["h"], -p["h"]).to(P.dtype)
        if "c" in p:
            P = P + torch.tensor(p["c"], device=DEV, dtype=torch.float32)
        out.append(P)
    return torch.cat(out), prims, origin, r_root


def _samples(scene, n, depth, seed):
    """Noisy surface samples and their radii."""
    P, prims, origin, r_root = _points(scene, n, seed)
    g = _gen(seed + 7_000_003)
    half = r_root / (1 << depth)
    return P + 1.5 * half * torch.randn(P.shape, generator=g, device=DEV), _radii(n, half, depth, g), prims, origin, r_root


def _radii(n, half, depth, g):
    """Most samples ask for cubes at `depth` and `depth` - 1; 3 % (silhouettes,
    isolated pixels) for a coarser one, which fills every level down to 2."""
    r = 1.5 * half * torch.exp(0.45 * torch.randn(n, generator=g, device=DEV))
    far = torch.rand(n, generator=g, device=DEV) < 0.03
    return torch.where(far, r * torch.exp2((depth - 2) * torch.rand(n, generator=g, device=DEV)), r)


def _taken(key, rc, n):
    """The first n cubes in Morton order, so that a case has one size whatever the seed."""
    if len(key) < n:
        raise ValueError(f"the samples made {len(key)} cubes: {n} are wanted")
    return key[:n].contiguous(), rc[:n].contiguous()


def _octree(case, seed, balanced=True):
    """(key = code | depth, r_c) of the merged and 2:1-balanced cubes, sorted."""
    P, r, prims, origin, r_root = _samples(case["scene"], case["samples"], case["depth"], seed)
    key, rc = S.cubes_from_samples(P, r, origin, r_root, case["depth"], torch)
    if balanced:
        key, rc = S.balance_2to1(key, rc, r_root, torch)
    return *_taken(key, rc, case["cubes"]), prims, origin, r_root


def _records(key, rc):
    """(n, 4) int32 device tensor of OctreeCube records."""
    code = key & ~31
    hi, lo = (code >> 32).to(torch.int32), (code & 0xFFFFFFFF)
    lo = torch.where(lo >= 1 << 31, lo - (1 << 32), lo).to(torch.int32)
    return torch.stack([hi, lo, rc.view(torch.int32), (key & 31).to(torch.int32)], 1).contiguous()


def _cube_array(rec):
    return rec.cpu().numpy().view(F.CUBE_DTYPE).reshape(-1)


def _centres(key, origin, r_root):
    code, d = key & ~31, key & 31
    cell = 2.0 * r_root / torch.exp2(d.float())
    xyz = [S._t_gather3(code >> a, torch) >> (21 - d) for a in range(3)]
    return torch.stack([o + (x.float() + 0.5) * cell for o, x in zip(origin, xyz)], 1)


def _distance(prims, p):
    """Signed distance of points to the union of the scene's primitives."""
    return torch.stack([S._sdf(q, p[:, 0], p[:, 1], p[:, 2], torch) for q in prims]).min(0).values


def _votes(key, rc, prims, origin, r_root, nbins, seed):
    """Histogram rows as ray-cast maps give them: 0..12 cameras see a cube, each
    votes for the bin of its noisy signed distance over 6 r_c; about 4 % of the
    cubes have no vote."""
    g = _gen(seed + 11)
    n = len(key)
    sd = _distance(prims, _centres(key, origin, r_root))
    seen = torch.randint(0, 13, (n,), generator=g, device=DEV)
    seen = torch.where(torch.rand(n, generator=g, device=DEV) < 0.04, 0, seen.clamp(min=1))
    h = torch.zeros((n, nbins), dtype=torch.int32, device=DEV)
    for k in range(12):
        a = ((sd + 0.5 * rc * torch.randn(n, generator=g, device=DEV)) / (6.0 * rc)).clamp(-1, 1)
        b = ((a + 1) * (nbins / 2)).long().clamp(max=nbins - 1)
        h.scatter_add_(1, b[:, None], (seen > k).to(torch.int32)[:, None])
    return h


def _rig(n, width, height):
    return S.sphere_rig(n, 4.0, width=width, height=height, half_fov_deg=25.0)


def _balls(seed):
    rng = np.random.default_rng(seed)
    return [(rng.uniform(-0.9, 0.9, 3), r) for r in (0.35, 0.4, 0.5, 0.6, 0.65)]


def _depth_of(cam, balls, sigma, seed):
    """Depth map (NaN where no surface) of a union of balls plus noise."""
    g = _gen(seed)
    Wd, H = cam["width"], cam["height"]
    v, u = torch.meshgrid(torch.arange(H, device=DEV, dtype=torch.float32),
                          torch.arange(Wd, device=DEV, dtype=torch.float32), indexing="ij")
    rt = np.asarray(cam["rt"], np.float64)
    d = [(u - cam["cx"]) / cam["fx"], (v - cam["cy"]) / cam["fy"], torch.ones_like(u)]
    best = torch.full_like(u, float("inf"))
    for c, r in balls:
        o = (rt[:3, :3].T @ (np.asarray(c) - rt[:3, 3])).tolist()  # centre in camera space
        b = d[0] * o[0] + d[1] * o[1] + d[2] * o[2]
        a = d[0] * d[0] + d[1] * d[1] + 1.0
        disc = b * b - a * (o[0] ** 2 + o[1] ** 2 + o[2] ** 2 - r * r)
        z = (b - torch.sqrt(disc.clamp(min=0))) / a
        best = torch.minimum(best, torch.where((disc > 0) & (z > 0), z, torch.full_like(z, float("inf"))))
    best = best + sigma * torch.randn(best.shape, generator=g, device=DEV)
    return torch.where(torch.isfinite(best), best, torch.full_like(best, float("nan")))


def _ball_cubes(case, balls, seed):
    """Balanced cubes around the balls' surfaces, as the maps' samples give them."""
    g = _gen(seed + 3)
    n, depth = case["samples"], case["depth"]
    r_root, origin = 2.0, (-2.0, -2.0, -2.0)
    w = torch.tensor([r * r for _, r in balls], device=DEV).cumsum(0)
    k = torch.bucketize(torch.rand(n, generator=g, device=DEV) * w[-1], w).clamp(max=len(balls) - 1)
    d = torch.randn((n, 3), generator=g, device=DEV)
    c = torch.tensor(np.array([b[0] for b in balls]), device=DEV, dtype=torch.float32)
    r = torch.tensor([b[1] for b in balls], device=DEV, dtype=torch.float32)
    half = r_root / (1 << depth)
    P = c[k] + r[k, None] * d / d.norm(dim=1, keepdim=True)
    P = P + 1.5 * half * torch.randn((n, 3), generator=g, device=DEV)
    rx = _radii(n, half, depth, g)
    key, rc = S.cubes_from_samples(P, rx, origin, r_root, depth, torch)
    key, rc = S.balance_2to1(key, rc, r_root, torch)
    return *_taken(key, rc, case["cubes"]), origin, r_root


def _pyramid(base):
    """All levels of a map, concatenated: 2x2 means of the finite, positive texels."""
    levels, x = [base.reshape(-1)], base
    for _ in range(12):
        h, w = x.shape
        if w <= 1 or h <= 1:
            break
        x = x[: h // 2 * 2, : w // 2 * 2].reshape(h // 2, 2, w // 2, 2)
        ok = torch.isfinite(x) & (x > 0)
        cnt = ok.sum((1, 3))
        x = torch.where(ok, x, torch.zeros_like(x)).sum((1, 3)) / cnt
        x = torch.where(cnt > 0, x, torch.full_like(x, float("nan")))
        levels.append(x.reshape(-1))
    return torch.cat(levels)


def _pinned(shape, dtype):
    """A zeroed numpy array in page-locked host memory."""
    return torch.zeros(shape, dtype=dtype).pin_memory().numpy()


def _pin(a):
    """The array's copy in page-locked host memory."""
    t = torch.from_numpy(np.ascontiguousarray(a).view(np.uint8).reshape(-1)).pin_memory()
    return t.numpy().view(a.dtype).reshape(a.shape)


def _rand_seed(seed):
    return int(seed) * 1_000_003 % (1 << 31)


# -------------------------------------------------------------------- prepare ---

def prepare(case, seed):
    seed = _rand_seed(seed)
    return _PREPARE[case["kind"]](case, seed) | {"case": case}


def _solve_inputs(case, seed):
    """Device cubes (n, 4) int32 and histograms (n, nbins) int32, host leaves or None."""
    rng = np.random.default_rng(seed)
    if case["scene"] == "octree":
        cubes = S.random_octree(rng, 2, case["depth"], case["cubes"])
        h = S.random_histograms(rng, len(cubes), case["nbins"])
        rec = torch.from_numpy(cubes.view(np.int32).reshape(-1, 4).copy()).to(DEV)
        hist = torch.from_numpy(h.view(np.int32)).to(DEV)
    else:
        key, rc, prims, origin, r_root = _octree(case, seed)
        rec = _records(key, rc)
        hist = _votes(key, rc, prims, origin, r_root, case["nbins"], seed)
        cubes = _cube_array(rec) if case["where"] == "host" or case["mode"] != "inmem" else None
    leaves = W.chunk_leaves(cubes, case.get("chunks", 1), rng) if case["mode"] != "inmem" else None
    return rec, hist, cubes, leaves


def _prep_solve(case, seed):
    rec, hist, cubes, leaves = _solve_inputs(case, seed)
    prm = api.TGVParams(alpha0=case["alpha0"], alpha1=case["alpha1"], iters=case["iters"], tol=case["tol"])
    if case["where"] == "host":
        return dict(cubes=cubes, hists=hist.cpu().numpy().view(np.uint32), leaves=leaves, prm=prm)
    out = torch.empty((len(rec), 13), dtype=torch.float32, device=DEV)
    return dict(cubes=rec, hists=hist, out=out, leaves=leaves, prm=prm)


def _prep_hist_host(case, seed):
    balls = _balls(seed)
    rig = _rig(case["maps"], case["width"], case["height"])
    maps = [_depth_of(c, balls, 0.003, seed + i).cpu().numpy() for i, c in enumerate(rig)]
    key, rc, origin, r_root = _ball_cubes(case, balls, seed)
    return dict(cubes=_cube_array(_records(key, rc)), cams=[W.camera(c) for c in rig], maps=maps, origin=origin,
                r_root=r_root)


def _prep_hist_dev(case, seed):
    balls = _balls(seed)
    rig = _rig(case["maps"], case["width"], case["height"])
    pyr = [_pyramid(_depth_of(c, balls, 0.003, seed + i)) for i, c in enumerate(rig)]
    off = np.concatenate([[0], np.cumsum([len(p) for p in pyr])]).astype(np.int64)
    key, rc, origin, r_root = _ball_cubes(case, balls, seed)
    cams = [W.camera(c) for c in rig]
    rec = _records(key, rc)
    out = torch.empty((len(rec), case["nbins"]), dtype=torch.int32, device=DEV)
    torch.cuda.synchronize()
    return dict(cubes=rec, cams=(N.Camera * len(cams))(*cams), tex=torch.cat(pyr), off=off, out=out,
                origin=np.asarray(origin, np.float32), r_root=r_root)


def _prep_stage1(case, seed):
    rng = np.random.default_rng(seed)
    cam = S.sphere_rig(64, 4.5 * rng.uniform(0.9, 1.1), width=case["width"], height=case["height"])[rng.integers(64)]
    depth = _pin(_depth_of(cam, _balls(seed), case["sigma"], seed).cpu().numpy())
    m = N.DepthMapS()
    m.fx, m.fy, m.cx, m.cy = cam["fx"], cam["fy"], cam["cx"], cam["cy"]
    m.rt[:] = [float(x) for x in cam["rt"].reshape(16)]
    m.width, m.height = case["width"], case["height"]
    m.depths = depth.ctypes.data_as(C.POINTER(C.c_float))
    return dict(map=m, depth=depth, origin=np.float32([-2, -2, -2]), r_root=2.0,
                out=_pinned((depth.size, 4), torch.int32).view(F.CUBE_DTYPE).reshape(-1))


def _merge_lists(case, seed):
    """Each list holds the code-sorted, unmerged cubes of one view: the samples
    of the half of the surface that faces it."""
    out = []
    P0, r0, _, origin, r_root = _samples("torus", 2 * case["per_list"], case["depth"], seed)
    for k in range(case["lists"]):
        d = torch.randn(3, generator=_gen(seed + 100 + k), device=DEV)
        m = (P0 @ d).argsort(descending=True)[: case["per_list"]]
        P = P0[m] + 0.3 * r_root / (1 << case["depth"]) * torch.randn((len(m), 3), generator=_gen(seed + 300 + k),
                                                                     device=DEV)
        r = r0[m]
        n = ((P - torch.tensor(origin, device=DEV)) / (2 * r_root)).clamp(0, 1 - 1e-6)
        dd = S.cube_depth_for_radius(r, r_root, case["depth"], torch)
        ix = (n * torch.exp2(dd.float())[:, None]).long() << (21 - dd)[:, None]
        key = S._t_encode(ix[:, 0], ix[:, 1], ix[:, 2], torch) | dd
        order = (key & ~31).sort(stable=True).indices  # by code; equal codes in sample order
        out.append(_cube_array(_records(key[order], r[order])))
    return out


def _prep_merge(case, seed):
    lists = [_pin(c) for c in _merge_lists(case, seed)]
    ns = np.array([len(c) for c in lists], np.int64)
    return dict(lists=lists, ptrs=(C.c_void_p * len(lists))(*[c.ctypes.data for c in lists]), ns=ns,
                out=_pinned((int(ns.sum()), 4), torch.int32).view(F.CUBE_DTYPE).reshape(-1))


def _prep_balance(case, seed):
    key, rc, _, _, r_root = _octree(case, seed, balanced=False)
    return dict(cubes=_pin(_cube_array(_records(key, rc))), r_root=r_root,
                out=_pinned((3 * len(key), 4), torch.int32).view(F.CUBE_DTYPE).reshape(-1))


def _prep_surface(case, seed):
    key, rc, prims, origin, r_root = _octree(case, seed)
    g = _gen(seed + 5)
    sd = _distance(prims, _centres(key, origin, r_root))
    st = 0.02 * torch.randn((len(key), 13), generator=g, device=DEV)
    st[:, 0] = (sd / (6 * rc) + 0.01 * torch.randn(len(key), generator=g, device=DEV)).clamp(-1, 1)
    has = (torch.rand(len(key), generator=g, device=DEV) > 0.04).to(torch.uint8)
    n = len(key)
    return dict(cubes=_pin(_cube_array(_records(key, rc))), state=_pin(st.cpu().numpy()), has=_pin(has.cpu().numpy()),
                origin=np.asarray(origin, np.float32), r_root=r_root, verts=np.zeros((5 * n, 3), np.float32),
                faces=np.zeros((3 * n, 3), np.uint32), normals=np.zeros((5 * n, 3), np.float32))


def _prep_mlp_infer(case, seed):
    rng = np.random.default_rng(seed)
    key, rc, prims, origin, r_root = _octree(case, seed)
    rec = _records(key, rc)
    hist = _votes(key, rc, prims, origin, r_root, case["nbins"], seed)
    leaves = W.chunk_leaves(_cube_array(rec), case["chunks"], rng)
    u = torch.empty(len(rec), dtype=torch.float32, device=DEV)
    torch.cuda.synchronize()
    return dict(cubes=rec, hists=hist, leaves=leaves, u=u, mlp=WS.WarmStartMLP(case["nbins"], seed=seed))


def _mlp_rows(case, seed):
    """Feature rows (bf16 bit patterns) and targets of a training set."""
    g = _gen(seed)
    n, nb = case["rows"], case["nbins"]
    X = torch.zeros((n, 16), device=DEV)
    h = torch.rand((n, nb), generator=g, device=DEV).pow(6)
    X[:, :nb] = h / h.sum(1, keepdim=True)
    X[:, nb] = torch.randint(2, 9, (n,), generator=g, device=DEV) / 21.0
    X[:, nb + 1: nb + 4] = torch.rand((n, 3), generator=g, device=DEV)
    X[:, nb + 4] = -1 + (torch.randint(0, nb, (n,), generator=g, device=DEV) + 0.5) / (nb / 2)
    X = X.to(torch.bfloat16)
    t = 0.1 * torch.sin(3 * X[:, nb + 4].float()) + 0.05 * torch.randn(n, generator=g, device=DEV)
    return X, t


def _prep_mlp_grad(case, seed):
    X, t = _mlp_rows(case, seed)
    return dict(X=X.view(torch.int16).cpu().numpy().view(np.uint16), t=t.cpu().numpy(),
                mlp=WS.WarmStartMLP(case["nbins"], seed=seed))


_PREPARE = dict(solve=_prep_solve, hist_host=_prep_hist_host, hist_dev=_prep_hist_dev, stage1=_prep_stage1,
                merge=_prep_merge, balance=_prep_balance, surface=_prep_surface, mlp_infer=_prep_mlp_infer,
                mlp_grad=_prep_mlp_grad)


# ------------------------------------------------------------------------ run ---

def _state_out(o):
    return {k: o[k] for k in ("u", "v", "p", "q")}


def _cubes_out(c, n):
    """The program's whole record buffer (zero beyond the n records written)."""
    w = c.view(np.int32).reshape(-1, 4)
    return dict(n=n, hi=w[:, 0], lo=w[:, 1], depth=w[:, 3], r_c=c["r_c"])


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "solve":
        if case["where"] == "host":
            if case["mode"] == "inmem" and case["tol"] == 0.0:
                return _state_out(api.tgv_minimize(s["cubes"], s["hists"], params=s["prm"]))
            return _state_out(api.tgv_solve(s["cubes"], s["hists"], s["leaves"], case["mode"], s["prm"])[0])
        api.tgv_solve_device(s["cubes"], s["hists"], s["out"], s["leaves"], case["mode"], s["prm"])
        o = s["out"]
        return dict(u=o[:, 0], v=o[:, 1:4], p=o[:, 4:7], q=o[:, 7:])
    if kind == "hist_host":
        return api.compute_histograms_from_maps(s["cubes"], s["cams"], s["maps"], s["origin"], s["r_root"],
                                                case["nbins"]).view(np.int32)
    if kind == "hist_dev":
        ctx = api.context()
        ctx.check(ctx.lib.tgvg_compute_histograms_dev(
            ctx.h, s["cubes"].data_ptr(), len(s["cubes"]), s["cams"], len(s["cams"]), s["tex"].data_ptr(),
            s["off"].ctypes.data, s["origin"].ctypes.data, s["r_root"], case["nbins"], s["out"].data_ptr()),
            "compute_histograms")
        return s["out"]
    if kind in ("stage1", "merge", "balance"):
        ctx, n = api.context(), C.c_int64()
        out = (s["out"].ctypes.data, len(s["out"]), C.byref(n))
        if kind == "stage1":
            ctx.check(ctx.lib.tgvg_build_cubes(ctx.h, C.byref(s["map"]), s["origin"].ctypes.data, s["r_root"], *out),
                      "tgvg_build_cubes")
        elif kind == "merge":
            ctx.check(ctx.lib.tgvg_merge_cubes(ctx.h, s["ptrs"], s["ns"].ctypes.data, len(s["ns"]), *out),
                      "tgvg_merge_cubes")
        else:
            ctx.check(ctx.lib.tgvg_balance_cubes(ctx.h, s["cubes"].ctypes.data, len(s["cubes"]), s["r_root"], *out),
                      "tgvg_balance_cubes")
        return _cubes_out(s["out"], n.value)
    if kind == "surface":
        ctx, h = api.context(), C.c_void_p()
        ctx.check(ctx.lib.tgvg_extract_surface(ctx.h, s["cubes"].ctypes.data, s["state"].ctypes.data, len(s["cubes"]),
                                               s["has"].ctypes.data, s["origin"].ctypes.data, s["r_root"], 1,
                                               C.byref(h)), "tgvg_extract_surface")
        nv, nf = C.c_int64(), C.c_int64()
        ctx.check(ctx.lib.tgvg_mesh_size(h, C.byref(nv), C.byref(nf), None), "tgvg_mesh_size")
        if nv.value > len(s["verts"]) or nf.value > len(s["faces"]):
            raise ValueError("the mesh does not fit the program's buffers")
        ctx.check(ctx.lib.tgvg_mesh_read(h, s["verts"].ctypes.data, s["faces"].ctypes.data, s["normals"].ctypes.data),
                  "tgvg_mesh_read")
        ctx.lib.tgvg_mesh_free(h)
        return dict(verts=s["verts"], faces=s["faces"].view(np.int32), normals=s["normals"], sizes=[nv.value, nf.value])
    if kind == "mlp_infer":
        m, lv = s["mlp"], s["leaves"]
        m.ctx.check(m.lib.tgvg_mlp_warm_start_dev(m.ctx.h, m.h, s["cubes"].data_ptr(), s["hists"].data_ptr(),
                                                  len(s["cubes"]), case["nbins"], lv.ctypes.data, len(lv),
                                                  s["u"].data_ptr()), "tgvg_mlp_warm_start")
        return s["u"]
    loss, g = s["mlp"].grad(s["X"], s["t"])
    return dict(loss=loss, grad=g)


# ----------------------------------------------------------------------- work ---

L2_BYTES = 129e6


def work(case):
    """Each input read once and each output written once.  An iteration of a
    level whose state (100 B a cube) is larger than the L2 cannot keep it on
    chip: it reads and writes u, v, the bars, p, q and reads the data term and
    the six neighbour indices once (168 B a cube).  About 130 operations per
    cube and iteration; a tolerance-stopped solve is counted at its cap only
    where levels reach it, taken here as one iteration in four."""
    k = case["kind"]
    n = case.get("cubes", 0)
    if k == "solve":
        # about 60 % of a generated octree's cubes are on its last level, 30 % on the one before
        lv = [0.6 * n, 0.3 * n, 0.1 * n]
        it = case["iters"] * (0.25 if case["tol"] > 0 else 1.0)
        b = n * (16 + 4 * case["nbins"] + 52) + sum(168 * c * it for c in lv if 100 * c > L2_BYTES)
        return dict(bytes=b, flops=130.0 * n * it)
    if k in ("hist_host", "hist_dev"):
        px = case["maps"] * case["width"] * case["height"]
        # projecting a pair: 7 multiplies and adds each for x, y, z, four divisions, level, texel and bin
        return dict(bytes=n * (16 + 4 * case["nbins"]) + 4 * px * (1 if k == "hist_host" else 4 / 3),
                    flops=45.0 * n * case["maps"])
    if k == "stage1":
        px = case["width"] * case["height"]
        return dict(bytes=px * 4 + 0.22 * px * 16, flops=120.0 * px)  # about 22 % of the pixels see a surface
    if k == "merge":
        n = case["lists"] * case["per_list"]  # about half of the entries are a cube of their own
        return dict(bytes=16 * n + 16 * 0.5 * n, flops=10.0 * n)
    if k == "balance":
        return dict(bytes=16 * n + 16 * 1.3 * n, flops=60.0 * n)
    if k == "surface":
        # a third of the cubes own a sign change: about one vertex with its normal and two triangles each
        return dict(bytes=n * (16 + 4 + 1) + n / 3 * (24 * 2 + 24), flops=100.0 * n)
    if k == "mlp_infer":
        return dict(bytes=n * (16 + 4 * case["nbins"] + 4), flops=n * 2.0 * (16 * 64 + 64 * 64 + 64))
    return dict(bytes=case["rows"] * 36, flops=case["rows"] * 3 * 2.0 * (16 * 64 + 64 * 64 + 64))


# ---------------------------------------------------------------------- exact ---

def exact(case, seed):
    seed = _rand_seed(seed)
    k = case["kind"]
    if k == "solve":
        # streaming and tolerance-stopped solves run thousands of iterations per level: far over 20 s here
        if case["mode"] != "inmem" or case["tol"] > 0:
            return None
        return _exact_solve(case, seed)
    if k == "merge":
        return _exact_merge(_merge_lists(case, seed))
    if k == "mlp_infer":
        s = _prep_mlp_infer(case, seed)
        return _exact_warm_start(s, case["nbins"])
    if k == "mlp_grad":
        X, t = _mlp_rows(case, seed)
        return _exact_grad(WS.WarmStartMLP(case["nbins"], seed=seed).get_params(), X, t)
    # histograms are whole numbers; Stage 1's and the balance's cube order and the surface's vertex
    # numbering follow float32 decisions cube by cube, so 64-bit values have no place beside them
    return None


def _exact_solve(case, seed):
    """The in-memory solve in 64 bits (reference src/tgv.cpp): levels coarse to
    fine, per iteration p and q from the bars, then u and v, then the bars."""
    rec, hist, _, _ = _solve_inputs(case, seed)
    n, nb = len(rec), case["nbins"]
    key = (rec[:, 0].long() << 32) | (rec[:, 1].long() & 0xFFFFFFFF)
    dep = rec[:, 3].long()
    cnt = hist.long()
    tot = cnt.sum(1)
    kk = (cnt.cumsum(1) * 2 >= tot[:, None]).int().argmax(1)
    med = torch.where(tot > 0, -1.0 + (kk.double() + 0.5) / (nb / 2.0), torch.zeros((), device=DEV, dtype=torch.float64))
    shrink = 0.25 * tot.double()
    # code -> largest index
    order = torch.sort(key, stable=True)
    skey, sidx = order.values, order.indices

    def find(k, ok):
        p = torch.searchsorted(skey, k, right=True) - 1
        hit = ok & (p >= 0)
        p = p.clamp(min=0)
        return torch.where(hit & (skey[p] == k), sidx[p], torch.full_like(p, -1))

    par_code = S._t_anc(key, (dep - 1).clamp(min=0), torch)
    par = find(par_code, dep > 0)
    nbr = []
    for f in range(6):
        c, ok = S._t_face(key, dep, f, torch)
        j = find(c, ok)
        pj = find(S._t_anc(c, (dep - 1).clamp(min=0), torch), ok & (dep > 0))
        nbr.append(torch.where(j >= 0, j, pj))
    f64 = dict(dtype=torch.float64, device=DEV)
    uv = torch.zeros((4, n), **f64)
    uv[0] = med
    bar = uv.clone()
    p, q = torch.zeros((3, n), **f64), torch.zeros((6, n), **f64)
    a0, a1 = float(np.float32(case["alpha0"])), float(np.float32(case["alpha1"]))
    first = int(dep.min())
    for d in range(first, int(dep.max()) + 1):
        idx = (dep == d).nonzero()[:, 0]
        if len(idx) == 0:
            continue
        if d > first:
            j = par[idx]
            uv[:, idx] = torch.where(j >= 0, uv[:, j.clamp(min=0)], uv[:, idx])
            p[:, idx] = 0
            q[:, idx] = 0
        x = uv[:, idx].clone()
        bar[:, idx] = x
        P, Q = torch.zeros((3, len(idx)), **f64), torch.zeros((6, len(idx)), **f64)
        p[:, idx], q[:, idx] = P, Q
        pos = torch.full((n,), -1, dtype=torch.long, device=DEV)
        pos[idx] = torch.arange(len(idx), device=DEV)
        m = len(idx)

        def split(j):
            """(index into [this level | other cubes' fixed values | zero], those cubes)"""
            own = j >= 0
            loc = torch.where(own, pos[j.clamp(min=0)], torch.full_like(j, -1))
            oth = own & (loc < 0)
            cub = j[oth]
            ind = loc.clone()
            ind[oth] = m + torch.arange(len(cub), device=DEV)
            return ind, cub

        me = torch.arange(m, device=DEV)
        fwd, bwd = [], []
        for a in range(3):
            ind, cub = split(nbr[2 * a][idx])
            fwd.append((torch.where(ind < 0, me, ind), bar[:, cub].clone()))
            ind, cub = split(nbr[2 * a + 1][idx])
            fixed = torch.cat([p[:, cub], q[:, cub]])
            z = m + len(cub)
            bwd.append((torch.where(ind < 0, torch.full_like(ind, z), ind), fixed))
        B, sh, md = x.clone(), shrink[idx], med[idx]
        zero = torch.zeros((9, 1), **f64)
        empty = tot[idx] == 0
        for _ in range(case["iters"]):
            g = [torch.cat([B, fx], 1)[:, i] for i, fx in fwd]
            P = P + 0.25 * torch.stack([g[a][0] - B[0] - B[a + 1] for a in range(3)])
            nrm = P.square().sum(0).sqrt()
            P = torch.where(nrm > a1, P * (a1 / nrm.clamp(min=1e-300)), P)
            e = [g[0][1] - B[1], g[1][2] - B[2], g[2][3] - B[3],
                 0.5 * (g[1][1] - B[1] + g[0][2] - B[2]), 0.5 * (g[2][1] - B[1] + g[0][3] - B[3]),
                 0.5 * (g[2][2] - B[2] + g[1][3] - B[3])]
            Q = Q + 0.25 * torch.stack(e)
            nrm = Q.square().sum(0).sqrt()
            Q = torch.where(nrm > a0, Q * (a0 / nrm.clamp(min=1e-300)), Q)
            PQ = torch.cat([P, Q])
            h = [torch.cat([PQ, fx, zero], 1)[:, i] for i, fx in bwd]
            z = x[0] + 0.25 * ((P[0] - h[0][0]) + (P[1] - h[1][1]) + (P[2] - h[2][2]))
            df = z - md
            un = torch.where(df > sh, z - sh, torch.where(df < -sh, z + sh, md))
            un = torch.where(empty, z, un)
            dq = [(Q[0] - h[0][3]) + (Q[3] - h[1][6]) + (Q[4] - h[2][7]),
                  (Q[3] - h[0][6]) + (Q[1] - h[1][4]) + (Q[5] - h[2][8]),
                  (Q[4] - h[0][7]) + (Q[5] - h[1][8]) + (Q[2] - h[2][5])]
            new = torch.stack([un] + [x[a + 1] + 0.25 * (P[a] + dq[a]) for a in range(3)])
            B = 2 * new - x
            x = new
        uv[:, idx], bar[:, idx], p[:, idx], q[:, idx] = x, B, P, Q
    t = lambda v: v.T.contiguous()  # noqa: E731
    return dict(u=uv[0], v=t(uv[1:]), p=t(p), q=t(q))


def _exact_merge(lists):
    c = np.concatenate(lists)
    key = (c["hi"].astype(np.uint64) << np.uint64(32)) | c["lo"].astype(np.uint64)
    c = c[np.argsort(key, kind="stable")]
    start = np.ones(len(c), bool)
    start[1:] = (c["hi"][1:] != c["hi"][:-1]) | (c["lo"][1:] != c["lo"][:-1]) | (c["depth"][1:] != c["depth"][:-1])
    s = np.flatnonzero(start)
    r = np.add.reduceat(c["r_c"].astype(np.float64), s) / np.diff(np.append(s, len(c)))
    full = np.zeros(len(c))
    full[: len(r)] = r
    return dict(n=None, hi=None, lo=None, depth=None, r_c=full)


def _bf(x):
    return x.to(torch.bfloat16).double()


def _net(prm):
    w = torch.from_numpy(np.asarray(prm, np.float32)).to(DEV)
    i = np.cumsum([0, 16 * 64, 64, 64 * 64, 64, 64, 1])
    W1, b1, W2, b2, W3, b3 = (w[a:b] for a, b in zip(i, i[1:]))
    return _bf(W1).view(16, 64), b1.double(), _bf(W2).view(64, 64), b2.double(), _bf(W3), b3.double()


def _exact_warm_start(s, nb):
    """median + network with the features and hidden activations rounded to
    bf16 (the network's definition), everything else in 64 bits."""
    rec, h = s["cubes"], s["hists"].long()
    n = len(rec)
    tot = h.sum(1)
    kk = (h.cumsum(1) * 2 >= tot[:, None]).int().argmax(1)
    med = torch.where(tot > 0, -1.0 + (kk.double() + 0.5) / (nb / 2.0), torch.zeros((), device=DEV, dtype=torch.float64))
    key = (rec[:, 0].long() << 32) | (rec[:, 1].long() & 0xFFFFFFFF)
    d = rec[:, 3].long()
    lv = s["leaves"]
    first = torch.from_numpy(lv["first_idx"].astype(np.int64)).to(DEV)
    leaf = torch.searchsorted(first, torch.arange(n, device=DEV), right=True) - 1
    lkey = torch.from_numpy(F.cube_keys(lv).astype(np.int64)).to(DEV)[leaf]
    ld = torch.from_numpy(lv["depth"].astype(np.int64)).to(DEV)[leaf]
    X = torch.zeros((n, 16), dtype=torch.float64, device=DEV)
    X[:, :nb] = torch.where(tot[:, None] > 0, h.double() / tot.clamp(min=1)[:, None].double(), X[:, :nb])
    X[:, nb] = d.double() / 21
    for a in range(3):
        c, o = S._t_gather3(key >> a, torch).double(), S._t_gather3(lkey >> a, torch).double()
        X[:, nb + 1 + a] = ((c - o + 0.5 * torch.exp2((21 - d).double())) / torch.exp2((21 - ld).double())).clamp(0, 1)
    X[:, nb + 4] = med
    W1, b1, W2, b2, W3, b3 = _net(s["mlp"].get_params())
    h1 = _bf((_bf(X) @ W1 + b1).clamp(min=0))
    h2 = _bf((h1 @ W2 + b2).clamp(min=0))
    return med + h2 @ W3 + b3


def _exact_grad(prm, X, t):
    W1, b1, W2, b2, W3, b3 = _net(prm)
    X, t = X.double(), t.double()
    n = len(t)
    h1 = _bf((X @ W1 + b1).clamp(min=0))
    h2 = _bf((h1 @ W2 + b2).clamp(min=0))
    e = h2 @ W3 + b3 - t
    dy = 2 * e / n
    dz2 = torch.where(h2 > 0, dy[:, None] * W3, torch.zeros_like(h2))
    dz1 = torch.where(h1 > 0, dz2 @ W2.T, torch.zeros_like(h1))
    g = torch.cat([(X.T @ dz1).reshape(-1), dz1.sum(0), (h1.T @ dz2).reshape(-1), dz2.sum(0), h2.T @ dy, dy.sum()[None]])
    return dict(loss=(e.square().mean()).item(), grad=g)
