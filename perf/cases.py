"""The work this engine is measured on: builds, refits, edits, queries, adjoints and the
batched step, each through the calls a program makes (quarry.capi, quarry.torch,
quarry.pipeline).

Sizes are the benchmark's configurations (quarry.workloads) and the ranges below them down to
the smallest scenes the tests and examples use: scenes of about 1,000 to 1.3 M primitives,
1,000 to 1 M rays, 1,000 to 262,144 query points, batches of 4 to 48 uneven scenes.  Inputs
are made from the seed by the engine's own seeded generators.

Every tree, query and refit result is defined bit for bit (results do not depend on the tree,
the order or the schedule, and the builders are deterministic), so those cases compare
exactly; the adjoints are FP64 sums rounded to FP32 once.
"""
from __future__ import annotations

import ctypes
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "quarry-gpu_b200")
if PKG not in sys.path:
    sys.path.insert(0, PKG)

import quarry.torch as qtorch  # noqa: E402
from quarry import capi, pipeline, workloads  # noqa: E402

# ---------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------


def listed():
    return [
        # an interactive pick or a line-of-sight test: few rays on a small mesh, latency counts
        dict(name="rays_small", do="rays", scene="terrain", n=8192, q=2048, builder="lbvh",
             order="input", wide=False, occ=False),
        # the terrain benchmark: a height field scanned from above, LBVH, a million rays
        dict(name="rays_terrain", do="rays", scene="terrain", n=131072, q=1_000_000,
             builder="lbvh", order="coherent", wide=False, occ=True),
        # the city benchmark (the headline): diffuse light over a large static scene, SAH tree
        dict(name="rays_city", do="rays", scene="city", n=1_310_720, q=1_000_000, builder="sah",
             order="coherent", wide=False, occ=True),
        # the points benchmark: scan alignment, nearest neighbour of 20,000 points in a cloud
        dict(name="closest_cloud", do="closest", scene="volume", n=1_048_576, q=20_000,
             builder="lbvh", order="input", wide=False, lanes=4),
        # the city benchmark's queries: 8 nearest triangles of 20,000 points
        dict(name="knn_city", do="knn", scene="city", n=1_310_720, q=20_000, k=8, builder="sah",
             order="input", wide=False, lanes=8),
        # neighbourhoods in a noisy scan of a surface: single-pass radius query as CSR
        dict(name="radius_shell", do="radius", scene="sheet", n=1_048_576, q=20_000, found=24.0,
             builder="lbvh", order="coherent", wide=False, lanes=1, stash=True),
        # a cloud that arrives anew each frame: the fast builder
        dict(name="build_cloud", do="build", scene="volume", n=1_048_576, builder="lbvh"),
        # a static scene prepared for many rays: the binned SAH builder, 32 bins
        dict(name="build_city_sah", do="build", scene="city", n=1_310_720, builder="sah"),
        # an animated cloud: 1 % of the points move, the topology stays
        dict(name="refit_moved", do="refit", scene="volume", n=1_048_576, builder="lbvh",
             dirty=0.01, wide=False),
        # an edited level: 1 % of the triangles deleted, inserted, appended or moved
        dict(name="edit_city", do="edit", scene="city", n=1_310_720, builder="sah",
             fraction=0.01, mode="cluster"),
        # the adjoint benchmark: a fitting step over a million ellipsoids (build, query, backward)
        dict(name="fit_gaussians", do="grad", op="gaussian", n=1_048_576, q=262_144,
             order="coherent", wide=True),
        # the batch benchmark at 48 of its 256 scenes: every build and every query, one graph
        dict(name="batch_scenes", do="batch", terrains=24, clouds=24, tri_hi=500_000,
             point_hi=1_000_000, query_hi=100_000, k=16),
    ]


def _log(rng, lo, hi):
    """A whole number of [lo, hi], log-uniform, odd or even alike."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case of the same ranges: any of the operations, kinds, orders and layouts."""
    do = rng.choice(["rays", "closest", "knn", "radius", "build", "build", "refit", "edit",
                     "grad", "batch"])
    order = rng.choice(["input", "morton", "coherent"])
    wide = rng.random() < 0.3
    builder = rng.choice(["lbvh", "sah"])
    if do == "rays":
        return dict(do=do, scene=rng.choice(["terrain", "city"]), n=_log(rng, 1_000, 1_310_720),
                    q=_log(rng, 1_000, 1_000_000), builder=builder, order=order, wide=wide,
                    occ=rng.random() < 0.5)
    scene = rng.choice(["terrain", "city", "volume", "volume", "sheet", "gaussians"])
    n = _log(rng, 1_000, 1_048_576)
    if do in ("closest", "knn"):
        c = dict(do=do, scene=scene, n=n, q=_log(rng, 1_000, 100_000), builder=builder,
                 order=order, wide=wide, lanes=1 if wide else rng.choice([1, 1, 4, 8, 32]))
        if do == "knn":
            c["k"] = rng.choice([1, 4, 5, 8, 16, 32])
        return c
    if do == "radius":
        return dict(do=do, scene=rng.choice(["volume", "sheet"]), n=n, q=_log(rng, 1_000, 100_000),
                    found=round(math.exp(rng.uniform(math.log(2.0), math.log(64.0))), 2),
                    builder=builder, order=order, wide=wide, lanes=1, stash=rng.random() < 0.5)
    if do == "build":
        return dict(do=do, scene=scene, n=n, builder=builder)
    if do == "refit":
        return dict(do=do, scene=rng.choice(["volume", "sheet"]), n=n, builder=builder,
                    dirty=rng.choice([0.01, 0.1, 1.0]), wide=wide)
    if do == "edit":
        return dict(do=do, scene=rng.choice(["terrain", "city", "volume"]),
                    n=_log(rng, 20_000, 1_048_576), builder=builder,
                    fraction=rng.choice([0.002, 0.01]), mode=rng.choice(["cluster", "scatter"]))
    if do == "grad":
        return dict(do=do, op=rng.choice(["gaussian", "triangle", "ray"]), n=n,
                    q=_log(rng, 1_000, 262_144), order=order, wide=wide)
    s = _log(rng, 2, 20)
    return dict(do="batch", terrains=s, clouds=_log(rng, 2, 20), tri_hi=_log(rng, 10_000, 500_000),
                point_hi=_log(rng, 10_000, 1_000_000), query_hi=_log(rng, 4_000, 60_000), k=16)


# ---------------------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------------------
_KIND = {"terrain": "tri", "city": "tri", "volume": "point", "sheet": "point",
         "gaussians": "gauss"}
_ORDER = {"input": 0, "morton": capi.QK_ORDER_MORTON, "coherent": capi.QK_ORDER_COHERENT}
_LANES = {1: 0, 4: capi.QK_TUNE_SPLIT4, 8: capi.QK_TUNE_SPLIT8, 32: capi.QK_TUNE_SPLIT}


def _seed(seed):
    return 1 + int(seed) % 1_000_003


def _scene(name, n, seed):
    """(n', stride) host primitives: n' is n, or the generator's nearest size below it."""
    if name == "terrain":
        return workloads.terrain(max(2, math.isqrt(n // 2)), seed)
    if name == "city":
        return workloads.city(max(1, n // 10), seed)[0]
    if name == "gaussians":
        return workloads.gaussians(n, seed=seed)
    return workloads.point_cloud(name, n, seed)


def _bounds(name, items):
    if _KIND[name] == "tri":
        return workloads.bounds_of(items)
    p = items[:, :3]
    return p.min(axis=0), p.max(axis=0)


def _queries(name, items, q, seed):
    lo, hi = _bounds(name, items)
    return workloads.uniform_points(q, lo, hi, seed, 13)


def _rays(name, items, q, seed):
    lo, hi = workloads.bounds_of(items)
    if name == "terrain":
        return workloads.down_rays(q, float(lo[0]), float(hi[0]), float(lo[1]), float(hi[1]),
                                   100.0, seed)
    return workloads.cosine_rays(q, float(lo[0]), float(hi[0]), float(lo[1]), float(hi[1]),
                                 float(hi[2]) + 50.0, seed)


def _flags(case):
    f = _ORDER[case["order"]] | (capi.QK_WIDE if case["wide"] else 0)
    if case.get("occ") and not case["wide"]:
        f |= capi.QK_TUNE_HIGH_OCC
    if not case["wide"]:
        f |= _LANES[case.get("lanes", 1)]
        if case.get("stash"):
            f |= capi.QK_TUNE_STASH
    return f


def _tree(case, items):
    t = capi.DeviceTree(_KIND[case["scene"]], items, builder=case["builder"])
    if case.get("wide"):
        t.build_wide()
    return t


def _batch_scene(case, i, seed):
    """Scene i of a batch: the benchmark's size rule (log-uniform, drawn by the scene's index),
    contents from the seed.  A third of the queries each closest, kNN and radius at 0.02 x the
    diagonal; terrains get as many rays straight down."""
    tri = i < case["terrains"]
    n, q = workloads.batch_scene_sizes(
        i, (1_000, case["tri_hi"]) if tri else (4_000, case["point_hi"]),
        (1_000, case["query_hi"]))
    name, sd = ("terrain" if tri else "volume"), 1000 * seed + i
    items = _scene(name, n, sd)
    lo, hi = _bounds(name, items)
    pts = _queries(name, items, q, sd)
    a = q // 3
    r = 0.02 * float(np.linalg.norm(hi.astype(np.float64) - lo))
    rays = _rays(name, items, q, sd) if tri else np.zeros((0, 8), np.float32)
    return workloads.BatchScene(_KIND[name], items, pts[:a], pts[a:2 * a], pts[2 * a:],
                                float(np.float32(r)), rays)


def _lattice(tris):
    """(vertices, corner indices) of a terrain: its vertices sit on the unit lattice."""
    v = tris.reshape(-1, 3)
    cells = int(round(float(v[:, 0].max())))
    at = (np.rint(v[:, 1]) * (cells + 1) + np.rint(v[:, 0])).astype(np.int32)
    verts = np.zeros((int(at.max()) + 1, 3), np.float32)
    verts[at] = v
    return verts, at.reshape(-1, 3)


def _radius(case):
    """A radius that holds about `found` points: a ball of the cloud's volume (side 100) or a
    disc of its shell (radius 50)."""
    if case["scene"] == "volume":
        return (case["found"] * 1e6 * 3.0 / (4.0 * math.pi * case["n"])) ** (1.0 / 3.0)
    return math.sqrt(case["found"] * 4.0 * math.pi * 2500.0 / (math.pi * case["n"]))


def _shell_points(q, seed):
    """Query points near the noisy shell: other points of the same distribution, moved a little."""
    p = workloads.point_cloud("sheet", q, seed + 7)
    return p + workloads.uniform_points(q, [-0.5] * 3, [0.5] * 3, seed, 17)


def prepare(case, seed):
    do, sd = case["do"], _seed(seed)
    dev = capi.to_device
    if do == "batch":
        scenes = [_batch_scene(case, i, sd) for i in range(case["terrains"] + case["clouds"])]
        p = pipeline.BatchPipeline(scenes[:case["terrains"]], scenes[case["terrains"]:],
                                   k=case["k"])
        # launch shapes: the choices shipped for the benchmark's batch
        shapes = {("tri", "rays"): (256, 4, 0, 1), ("tri", "closest"): (256, 6, 16, 1),
                  ("tri", "knn"): (128, 6, 0, 5), ("tri", "radius"): (256, 8, 8, 8193),
                  ("point", "closest"): (256, 8, 8, 0), ("point", "knn"): (128, 6, 0, 5),
                  ("point", "radius"): (256, 6, 8, 8192)}
        for ph in p.phases:
            block, per_sm, short, flags = shapes[(ph.kind, ph.name)]
            ph.params = dict(ph.params, block=block, blocks_per_sm=per_sm, short_stack=short,
                             chunks_per_fetch=1, flags=flags, split=0)
        p.size_radius_outputs()
        for ph in p.phases:
            if ph.name == "radius":  # room for any scenes of these sizes
                n = np.array([len(sc.items) for sc in p.scenes[ph.kind]], np.float64)
                per = np.maximum(16.0, n * (0.006 if ph.kind == "tri" else 2e-4))
                ph.capacity = max(ph.capacity, int((ph.counts * per).sum()))
                ph.out = torch.zeros(ph.capacity, dtype=torch.int64, device="cuda")
        p.capture()
        return dict(do=do, pipe=p)
    if do == "grad":
        g = torch.Generator().manual_seed(sd)
        if case["op"] == "gaussian":
            it = workloads.gaussians(case["n"], seed=sd)
            pts = _queries("gaussians", it, case["q"], sd)
            parts = [pts, it[:, 0:3], it[:, 3:7], it[:, 7:10]]
            idx = None
        else:
            tris = workloads.terrain(max(2, math.isqrt(case["n"] // 2)), sd)
            verts, idx = _lattice(tris)
            idx = dev(idx)
            if case["op"] == "triangle":
                parts = [_queries("terrain", tris, case["q"], sd), verts]
            else:
                r = _rays("terrain", tris, case["q"], sd)
                parts = [r[:, 0:3], r[:, 3:6], verts]
        leaves = [dev(np.ascontiguousarray(a), np.float32).requires_grad_() for a in parts]
        w = (torch.rand(case["q"], generator=g) + 0.5).cuda()
        return dict(do=do, op=case["op"], leaves=leaves, idx=idx, w=w,
                    kw=dict(order=case["order"], wide=case["wide"]))
    items = _scene(case["scene"], case["n"], sd)
    kind = _KIND[case["scene"]]
    if do == "build":
        d = dev(items, np.float32)
        return dict(do=do, tree=capi.DeviceTree(kind, d, builder=case["builder"]))
    if do == "refit":
        tree = _tree(case, items)
        if case["dirty"] >= 1.0:
            moved = items + workloads.uniform_points(len(items), [-0.2] * 3, [0.2] * 3, sd, 19)
            return dict(do=do, tree=tree, ids=None, moved=dev(moved, np.float32))
        new, ids = workloads.coherent_motion(items, case["dirty"], seed=sd)
        return dict(do=do, tree=tree, ids=dev(ids, np.int32), moved=dev(new[ids], np.float32))
    if do == "edit":
        tree = _tree(case, items)
        new, dele, ins, mov = workloads.topology_edit(items, case["fraction"], case["mode"], sd)
        dst = capi.DeviceTree(kind, new)  # the arrays that receive the edited tree
        d, i, m = dev(dele, np.int32), dev(ins, np.int32), dev(mov, np.int32)
        appended = len(new) - len(items) + len(dele) - len(ins)
        extra = dev(np.concatenate([new[ins], new[len(new) - appended:]]), np.float32)
        moved = dev(new[mov], np.float32)
        e = capi.QkTopoEdit(d.data_ptr(), len(dele), i.data_ptr(), len(ins), appended,
                            m.data_ptr(), len(mov), extra.data_ptr(), moved.data_ptr())
        nb = capi.lib().qk_update_workspace_bytes(tree.kind, tree.n, dst.n, int(extra.shape[0]))
        ws = torch.empty(int(nb), dtype=torch.uint8, device="cuda")
        return dict(do=do, tree=tree, dst=dst, edit=e, ws=ws, keep=(d, i, m, extra, moved))
    tree = _tree(case, items)
    if do == "rays":
        return dict(do=do, tree=tree, rays=dev(_rays(case["scene"], items, case["q"], sd)),
                    flags=_flags(case))
    pts = dev(_queries(case["scene"], items, case["q"], sd), np.float32)
    if do == "radius":
        if case["scene"] == "sheet":
            pts = dev(_shell_points(case["q"], sd), np.float32)
        q, flags = case["q"], _flags(case)
        # a program that repeats the query keeps its buffers: offsets, keys and workspace
        nb = capi.lib().qk_radius_workspace_bytes(q, flags)
        return dict(do=do, tree=tree, pts=pts, r=_radius(case), flags=flags,
                    off=torch.empty(q + 1, dtype=torch.int32, device="cuda"),
                    keys=torch.zeros(int(3 * case["found"] * q) + 4096, dtype=torch.int64,
                                     device="cuda"),
                    ws=torch.empty(int(nb), dtype=torch.uint8, device="cuda"))
    return dict(do=do, tree=tree, pts=pts, k=case.get("k", 0), flags=_flags(case))


# ---------------------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------------------
def _arrays(t):
    return {name: t.arrays[name].view(torch.int32)
            for name in ("nodes", "items", "prim_ids", "parent", "depth_arr", "bnodes", "leaves",
                         "slot_of")}


def run(s):
    do = s["do"]
    if do == "rays":
        out = s["tree"].raycast(s["rays"], s["flags"])
        return {"t": out.view(torch.float32)[0::2], "hit": out.view(torch.int32)[1::2]}
    if do == "closest":
        out = s["tree"].closest(s["pts"], s["flags"])
        return {"dist2": out[:, 0].view(torch.float32), "id": out[:, 1]}
    if do == "knn":
        out = s["tree"].knn(s["pts"], s["k"], s["flags"])
        return {"dist2": out[..., 0].view(torch.float32), "id": out[..., 1]}
    if do == "radius":
        L, t, pts, ws, total = capi.lib(), s["tree"].t, s["pts"], s["ws"], ctypes.c_int64(0)
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        args = (ctypes.byref(t), pts.data_ptr(), len(pts), s["r"], s["off"].data_ptr())
        capi.check(L.qk_radius_count(*args, ctypes.byref(total), s["flags"], None, ws.data_ptr(),
                                     ws.numel(), stream), "qk_radius_count")
        if total.value > len(s["keys"]):
            raise RuntimeError(f"{total.value} keys, room for {len(s['keys'])}")
        capi.check(L.qk_radius_fill(*args, s["keys"].data_ptr(), s["flags"], ws.data_ptr(),
                                    ws.numel(), stream), "qk_radius_fill")
        return {"offsets": s["off"], "keys": s["keys"]}
    if do == "build":
        s["tree"].build()
        return _arrays(s["tree"])
    if do == "refit":
        t = s["tree"]
        if s["ids"] is None:
            t.refit(s["moved"])
        else:
            t.refit_dirty(s["ids"], s["moved"])
        out = {n: t.arrays[n].view(torch.int32) for n in ("nodes", "items", "bnodes", "leaves")}
        if "wide" in t.arrays:
            out["wide"] = t.arrays["wide"].view(torch.int32)
        return out
    if do == "edit":
        info = capi.QkTopoInfo()
        dst, ws = s["dst"], s["ws"]
        capi.check(capi.lib().qk_update_topology(
            ctypes.byref(s["tree"].t), ctypes.byref(dst.t), ctypes.byref(s["edit"]), 0, 32,
            ctypes.byref(info), ws.data_ptr(), ws.numel(),
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)), "qk_update_topology")
        if info.rebuild:
            dst.build()
        return _arrays(dst)
    if do == "grad":
        leaves, kw = s["leaves"], s["kw"]
        if s["op"] == "gaussian":
            d = qtorch.gaussian_distance(*leaves, **kw)
        elif s["op"] == "triangle":
            d = qtorch.triangle_distance(leaves[0], leaves[1], s["idx"], **kw)
        else:
            d, hit = qtorch.ray_hit_t(leaves[0], leaves[1], leaves[2], s["idx"], **kw)
        grads = torch.autograd.grad(d, leaves, grad_outputs=s["w"])
        return {"d": d.detach(), "grads": list(grads)}
    p = s["pipe"]
    p.replay()
    out = {}
    for ph in p.phases:
        out[f"{ph.kind}_{ph.name}"] = ph.out
        if ph.offsets is not None:
            out[f"{ph.kind}_{ph.name}_offsets"] = ph.offsets[: int(ph.counts.sum()) + 1]
    return out


# ---------------------------------------------------------------------------------------
# what a pass cannot do without, and how far results may differ
# ---------------------------------------------------------------------------------------
_ITEM = {"tri": 36, "point": 12, "gauss": 40}
_PAYLOAD = {"tri": 48, "point": 16, "gauss": 48}


def _tree_bytes(kind, n):
    """Every array of a tree of n primitives: canonical nodes, traversal nodes, payloads, items
    in leaf order, prim ids, inverse map, parents and depths."""
    return n * (64 + 64 + _PAYLOAD[kind] + _ITEM[kind] + 4 + 4 + 8 + 8)


def _walk_bytes(kind, n, q, leaves=1.0):
    """The least a batch of q queries reads of the tree: a root-to-leaf path of 64-byte nodes and
    `leaves` payloads each, and never more than the whole tree once."""
    path = 64.0 * math.log2(max(n, 2)) + leaves * _PAYLOAD[kind]
    return min(q * path, n * (64.0 + _PAYLOAD[kind]))


def work(case):
    do = case["do"]
    if do == "batch":
        m = lambda lo, hi: (hi - lo) / math.log(hi / lo)  # noqa: E731  mean of a log-uniform size
        nt, nc = m(1_000, case["tri_hi"]), m(4_000, case["point_hi"])
        q = m(1_000, case["query_hi"])
        t, c = case["terrains"], case["clouds"]
        b = t * nt * 36 + c * nc * 12 + t * _tree_bytes("tri", nt) + c * _tree_bytes("point", nc)
        b += t * q * 40 + (t + c) * q / 3 * (12 + 8 + 12 + 8 * case["k"] + 12 + 4 + 8 * 30)
        f = 300.0 * (2 * t + c) * q * math.log2(nt)
        return {"bytes": b, "flops": f}
    n = case["n"]
    if do == "grad":
        kind = "gauss" if case["op"] == "gaussian" else "tri"
        b = n * _ITEM[kind] + _tree_bytes(kind, n) + case["q"] * (2 * 24 + 12)
        b += n * 40 if kind == "gauss" else n * 18
        return {"bytes": b, "flops": case["q"] * (60.0 * math.log2(n) + 400.0)}
    kind = _KIND[case["scene"]]
    if do == "build":
        return {"bytes": n * _ITEM[kind] + _tree_bytes(kind, n),
                "flops": n * (60.0 if case["builder"] == "lbvh" else 40.0 * math.log2(n))}
    if do == "refit":
        m = n * case["dirty"]
        up = min(n, m * max(1.0, math.log2(n / m) if m < n else 1.0))
        b = m * 2 * _ITEM[kind] + up * (32 + 64 + 32 + 32) + m * _PAYLOAD[kind]
        return {"bytes": b, "flops": 12.0 * up}
    if do == "edit":
        return {"bytes": 2 * _tree_bytes(kind, n), "flops": 20.0 * n}
    q = case["q"]
    if do == "rays":
        return {"bytes": 40 * q + _walk_bytes(kind, n, q), "flops": q * (40.0 * math.log2(n) + 60)}
    k = 1 if do == "closest" else case.get("k", case.get("found", 1.0))
    b = q * (12 + 8 * k + (4 if do == "radius" else 0)) + _walk_bytes(kind, n, q, k)
    return {"bytes": b, "flops": q * (24.0 * math.log2(n) + 12.0 * k)}


def tolerance(case):
    if case["do"] == "grad":
        # FP64 terms and sums, one rounding to FP32 (half an ulp is 6e-8); distances are exact
        return {"rel": 2.5e-7, "max": 1e-5}
    return "exact"


# ---------------------------------------------------------------------------------------
# the same answers in 64 bits
# ---------------------------------------------------------------------------------------
_PAIRS = 3.0e10   # brute force up to this many (query, primitive) pairs
_CHUNK = 1 << 28  # pairs held at a time


def _point_triangle(p, tri):
    """Squared distance from points p (..., 3) to triangles tri (..., 9), in p's precision."""
    a, b, c = tri[..., 0:3], tri[..., 3:6], tri[..., 6:9]

    def edge(u, v):
        e = v - u
        t = (((p - u) * e).sum(-1) / (e * e).sum(-1).clamp_min(1e-300)).clamp(0.0, 1.0)
        return ((p - u - t[..., None] * e) ** 2).sum(-1)

    n = torch.linalg.cross(b - a, c - a)
    nn = (n * n).sum(-1).clamp_min(1e-300)
    h = ((p - a) * n).sum(-1)
    inside = torch.ones_like(h, dtype=torch.bool)
    for u, v in ((a, b), (b, c), (c, a)):
        inside &= (torch.linalg.cross(v - u, p - u) * n).sum(-1) >= 0
    border = torch.minimum(torch.minimum(edge(a, b), edge(b, c)), edge(c, a))
    return torch.where(inside & (nn > 1e-300), h * h / nn, border)


def _nearest(items, pts, k, kind):
    """(squared distances, ids) of the k nearest primitives by brute force in 64 bits."""
    items, pts = items.double(), pts.double()
    n = items.shape[0]
    k = min(k, n)
    # the expanded (pairs, 3) form is only for the triangles' few extra terms: smaller chunks
    per = max(1, (_CHUNK if kind == "point" else _CHUNK // 24) // n)
    ds, ids = [], []
    for i in range(0, len(pts), per):
        p = pts[i:i + per]
        if kind == "point":
            d = (p[:, None, 0] - items[None, :, 0]) ** 2
            d += (p[:, None, 1] - items[None, :, 1]) ** 2
            d += (p[:, None, 2] - items[None, :, 2]) ** 2
        else:
            d = _point_triangle(p[:, None, :], items[None, :, :])
        v, j = torch.topk(d, k, dim=1, largest=False)
        ds.append(v)
        ids.append(j)
    return torch.cat(ds), torch.cat(ids)


def _first_hits(tris, rays):
    """(t, id) of the first hit of each ray by brute force in 64 bits; t = inf, id = -1 on a miss."""
    tris, rays = tris.double(), rays.double()
    a, e1, e2 = tris[:, 0:3], tris[:, 3:6] - tris[:, 0:3], tris[:, 6:9] - tris[:, 0:3]
    ts, ids = [], []
    per = max(1, _CHUNK // 24 // tris.shape[0])
    for i in range(0, len(rays), per):
        o, d = rays[i:i + per, None, 0:3], rays[i:i + per, None, 3:6]
        pv = torch.linalg.cross(d.expand(-1, len(a), -1), e2[None].expand(len(o), -1, -1))
        det = (e1[None] * pv).sum(-1)
        s = o - a[None]
        u = (s * pv).sum(-1) / det
        qv = torch.linalg.cross(s, e1[None].expand_as(s))
        v = (d * qv).sum(-1) / det
        t = (e2[None] * qv).sum(-1) / det
        ok = (det != 0) & (u >= 0) & (v >= 0) & (u + v <= 1)
        ok &= (t >= rays[i:i + per, 6:7]) & (t <= rays[i:i + per, 7:8])
        t = torch.where(ok, t, torch.full_like(t, math.inf))
        best, j = t.min(dim=1)
        ts.append(best)
        ids.append(torch.where(torch.isfinite(best), j, -1))
    return torch.cat(ts), torch.cat(ids)


def _rotate_inv(quat, v):
    """v in the frame of the (normalised) xyzw quaternion."""
    q = quat / quat.norm(dim=-1, keepdim=True)
    u, w = -q[..., 0:3], q[..., 3:4]
    return v + 2.0 * torch.linalg.cross(u, torch.linalg.cross(u, v) + w * v)


def _ellipsoid_foot(y, s):
    """Unit direction u with s * u the point of the ellipsoid |x / s| = 1 nearest to y (outside),
    by bisection on the multiplier."""
    lo = torch.zeros_like(y[..., 0])
    hi = (s * y).norm(dim=-1)
    for _ in range(100):
        mid = 0.5 * (lo + hi)
        f = ((s * y / (s * s + mid[..., None])) ** 2).sum(-1)
        lo, hi = torch.where(f > 1, mid, lo), torch.where(f > 1, hi, mid)
    return s * y / (s * s + (0.5 * (lo + hi))[..., None])


def _ellipsoid_distance(p, mean, quat, scale):
    y = _rotate_inv(quat, p - mean)
    with torch.no_grad():
        out = ((y / scale) ** 2).sum(-1) > 1.0
        u = _ellipsoid_foot(y, scale)
    d = (y - scale * u).norm(dim=-1)  # stationary in u, so u's own dependence drops out
    return torch.where(out, d, torch.zeros_like(d))


def _nearest_ellipsoid(pts, it):
    """Index of the nearest ellipsoid of each point: the 64 of least (distance to the centre -
    largest axis) are measured in 64 bits."""
    mean, smax = it[:, 0:3].float(), it[:, 7:10].amax(dim=1).float()
    per = max(1, _CHUNK // len(it))
    k = min(64, len(it))
    ids = []
    for i in range(0, len(pts), per):
        p = pts[i:i + per]
        d = torch.cdist(p.float(), mean, compute_mode="donot_use_mm_for_euclid_dist")
        d -= smax
        j = torch.topk(d, k, dim=1, largest=False).indices
        g = it[j].double()
        e = _ellipsoid_distance(p.double()[:, None, :].expand(-1, k, -1), g[..., 0:3], g[..., 3:7],
                                g[..., 7:10])
        ids.append(j.gather(1, e.argmin(dim=1, keepdim=True))[:, 0])
    return torch.cat(ids)


def _exact_grad(case, seed):
    s = prepare(case, seed)
    x = [t.detach().double().requires_grad_() for t in s["leaves"]]
    if case["op"] == "gaussian":
        if len(x[1]) * float(len(x[0])) > 3.0e11:
            return None
        it = torch.cat(x[1:], dim=1).detach()
        j = _nearest_ellipsoid(x[0].detach(), it)
        d = _ellipsoid_distance(x[0], x[1][j], x[2][j], x[3][j])
    else:
        idx = s["idx"].long()
        if len(idx) * float(case["q"]) > _PAIRS:
            return None
        tris = x[-1].detach()[idx].reshape(-1, 9)
        if case["op"] == "triangle":
            _, j = _nearest(tris, x[0].detach(), 1, "tri")
            d2 = _point_triangle(x[0], x[1][idx[j[:, 0]]].reshape(-1, 9))
            d = torch.where(d2 > 0, d2, torch.ones_like(d2)).sqrt() * (d2 > 0)
        else:
            q = len(x[0])
            lim = torch.tensor([1e-6, math.inf], dtype=torch.float64, device="cuda").expand(q, 2)
            _, j = _first_hits(tris, torch.cat([x[0].detach(), x[1].detach(), lim], dim=1))
            tri = x[2][idx[j.clamp_min(0)]]
            n = torch.linalg.cross(tri[:, 1] - tri[:, 0], tri[:, 2] - tri[:, 0])
            t = ((tri[:, 0] - x[0]) * n).sum(-1) / (x[1] * n).sum(-1)
            d = torch.where(j >= 0, t, torch.full_like(t, math.inf))
            g = torch.autograd.grad(t, x, grad_outputs=s["w"].double() * (j >= 0))
            return {"d": d.detach(), "grads": list(g)}
    g = torch.autograd.grad(d, x, grad_outputs=s["w"].double())
    return {"d": d.detach(), "grads": list(g)}


def exact(case, seed):
    """Query distances, hits and adjoints in 64 bits by brute force; None where the outputs are
    packed trees or keys, or where brute force takes too long."""
    do = case["do"]
    if do == "grad":
        return _exact_grad(case, seed)
    if do not in ("rays", "closest", "knn") or case["n"] * float(case["q"]) > _PAIRS:
        return None
    kind = _KIND[case["scene"]]
    s = prepare(case, seed)
    items = s["tree"].items_scene
    if do == "rays":
        t, j = _first_hits(items, s["rays"])
        return {"t": torch.where(j >= 0, t, torch.zeros_like(t)), "hit": None}
    if kind == "gauss":
        return None
    d, _ = _nearest(items, s["pts"], max(1, case.get("k", 1)), kind)
    return {"dist2": d[:, 0] if do == "closest" else d, "id": None}
