"""Sizes at which the engine's tiled kernels can go wrong, bit for bit against the oracle: the
LBVH pass's blocks of 256 leaves, the radix sort's tiles of 4,096 keys, and the traversals'
forms (node arrays off a 32-byte boundary, every kNN table size, early-ended ellipsoid tests)."""
from __future__ import annotations

import numpy as np
import pytest

import oracle
from quarry import capi, workloads

pytestmark = pytest.mark.gpu


def _dev(a, dtype=np.float32):
    return capi.to_device(np.ascontiguousarray(a), dtype)


def _points(n, seed, distinct):
    """n points on `distinct` positions: few positions give runs of equal Morton codes, which only
    their indices order."""
    p = workloads.uniform_points(min(n, distinct), [0.0] * 3, [100.0] * 3, seed, 13)
    return np.ascontiguousarray(p[np.random.default_rng(seed).integers(0, len(p), n)])


@pytest.mark.parametrize("n", [2, 3, 31, 33, 255, 256, 257, 511, 513, 1025, 4096, 4097, 20001])
@pytest.mark.parametrize("distinct", [1, 7, 1 << 30])
def test_lbvh_block_edges(cuda, n, distinct):
    pts = _points(n, n, distinct)
    t, ref = capi.DeviceTree("point", pts), oracle.LBVH("point", pts)
    assert t.nodes_bytes().tobytes() == ref.nodes.tobytes()
    assert t.validate() == [0] * 8
    first = t.host("bnodes", np.uint8).copy()
    t.build()  # the arrival words are clean again
    assert t.nodes_bytes().tobytes() == ref.nodes.tobytes()
    assert np.array_equal(t.host("bnodes", np.uint8), first)


@pytest.mark.parametrize("sizes", [[2, 2, 2], [2, 257, 3, 1024, 1025, 5], [300] * 40])
def test_batched_lbvh_block_edges(cuda, sizes):
    scenes = [_points(n, 100 + i, 50) for i, n in enumerate(sizes)]
    b = capi.Batch("point", scenes)
    b.build()
    b.sync()
    for i, s in enumerate(scenes):
        v = b.view(i)
        assert v.nodes_bytes().tobytes() == oracle.LBVH("point", s).nodes.tobytes()
        assert v.validate() == [0] * 8


@pytest.mark.parametrize("n", [1, 4095, 4096, 4097, 8192, 70001])
@pytest.mark.parametrize("bits", [1, 8, 9, 16, 24, 30, 32])
@pytest.mark.parametrize("spread", [1, 3, 1 << 32])
def test_sort_tile_edges(cuda, n, bits, spread):
    rng = np.random.default_rng(n + bits)
    keys = (rng.integers(0, spread, n, dtype=np.uint64) & ((1 << bits) - 1)).astype(np.uint32)
    vals = rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32)
    k, v = capi.sort_pairs(_dev(keys.view(np.int32), np.int32), _dev(vals.view(np.int32), np.int32),
                           bits)
    o = np.argsort(keys, kind="stable")
    assert np.array_equal(k.cpu().numpy().view(np.uint32), keys[o])
    assert np.array_equal(v.cpu().numpy().view(np.uint32), vals[o])


def test_nodes_off_a_32_byte_boundary(cuda):
    """Traversal and 4-wide nodes on a 16-byte boundary: every schedule gives the same bits."""
    tris, _ = workloads.city(200, 3)
    lo, hi = workloads.bounds_of(tris)
    rays = _dev(workloads.cosine_rays(5000, float(lo[0]), float(hi[0]), float(lo[1]), float(hi[1]),
                                      float(hi[2]) + 50.0, 3))
    q = _dev(workloads.uniform_points(700, lo, hi, 3, 13))
    t = capi.DeviceTree("tri", tris)
    t.build_wide()
    flags = [0, capi.QK_TUNE_HIGH_OCC, capi.QK_ORDER_COHERENT, capi.QK_WIDE]
    want = [(t.raycast(rays, f).clone(), t.closest(q, f).clone(), t.knn(q, 8, f).clone())
            for f in flags]
    for name in ("bnodes", "wide"):
        a = t.arrays[name]
        moved = cuda.empty(a.numel() + 64, dtype=cuda.uint8, device="cuda")
        at = 16 - moved.data_ptr() % 32 if moved.data_ptr() % 32 < 16 else 48 - moved.data_ptr() % 32
        part = moved[at:at + a.numel()]
        assert part.data_ptr() % 32 == 16
        part.copy_(a)
        t.arrays[name] = part
        setattr(t.t, name, part.data_ptr())
    for f, (r, c, k) in zip(flags, want):
        assert cuda.equal(t.raycast(rays, f), r)
        assert cuda.equal(t.closest(q, f), c)
        assert cuda.equal(t.knn(q, 8, f), k)


@pytest.mark.parametrize("kind", ["tri", "point", "gauss"])
@pytest.mark.parametrize("k", [1, 3, 4, 5, 8, 11, 16, 17, 32])
def test_knn_every_table(cuda, kind, k):
    items = {"tri": lambda: workloads.terrain(12, 2), "point": lambda: _points(300, 5, 90),
             "gauss": lambda: workloads.gaussians(300, 0.5, 20.0, 4)}[kind]()
    c = items.reshape(len(items), -1)[:, :3]
    q = workloads.uniform_points(403, c.min(0) - 5, c.max(0) + 5, 9, 13)
    t, ref = capi.DeviceTree(kind, items), oracle.LBVH(kind, items)
    t.build_wide()
    want = ref.knn(q, k)
    for f in (0, capi.QK_WIDE, capi.QK_TUNE_SPLIT4, capi.QK_TUNE_SPLIT8, capi.QK_TUNE_SPLIT):
        assert np.array_equal(t.knn(_dev(q), k, f).cpu().numpy().view(np.uint32), want), f


@pytest.mark.parametrize("smin,smax", [(0.05, 1.0), (0.2, 8.0), (5.0, 5.0)])
def test_ellipsoid_tests_end_early_with_the_same_bits(cuda, smin, smax):
    """Needles, balls and plates: a test that stops once its distance is past the caller's limit
    never changes a result (closest, kNN and radius against tests run to the end)."""
    g = workloads.gaussians(1500, smin, smax, 8)
    q = workloads.uniform_points(1500, [-20.0] * 3, [120.0] * 3, 8, 13)
    t, ref = capi.DeviceTree("gauss", g), oracle.LBVH("gauss", g)
    t.build_wide()
    for f in (0, capi.QK_WIDE, capi.QK_TUNE_SPLIT):
        assert np.array_equal(t.closest(_dev(q), f).cpu().numpy().view(np.uint32), ref.closest(q)), f
        assert np.array_equal(t.knn(_dev(q), 6, f).cpu().numpy().view(np.uint32), ref.knn(q, 6)), f
        off, keys = t.radius(_dev(q), 9.0, f)
        woff, wkeys = ref.radius(q, 9.0)
        assert np.array_equal(off.cpu().numpy().astype(np.int64), woff), f
        assert np.array_equal(keys.cpu().numpy().view(np.uint64), wkeys), f


@pytest.mark.parametrize("thin", [1e-12, 6e-20, 5e-20, 1e-20, 1e-22, 1e-40])
@pytest.mark.parametrize("axes", [1, 2])
def test_ellipsoids_with_a_very_short_axis(cuda, thin, axes):
    """Axes whose squares are subnormal or zero, queries nearer to a centre than the longest axis
    (the iteration then starts at t = 0, where 1 / axis^2 overflows) and farther away: the oracle's
    results, which its brute force confirms do not depend on the visit order."""
    g = workloads.gaussians(300, 5.0, 20.0, 8)
    for i in range(len(g)):
        for a in range(axes if i % 3 else 0):  # a third keeps its axes
            g[i, 7 + (i + a) % 3] = thin
    q = np.concatenate([workloads.uniform_points(500, [-20.0] * 3, [120.0] * 3, 8, 13),
                        g[:200, :3] + workloads.uniform_points(200, [-3.0] * 3, [3.0] * 3, 9, 13)])
    t, ref = capi.DeviceTree("gauss", g), oracle.LBVH("gauss", g)
    t.build_wide()
    closest, knn = ref.closest(q), ref.knn(q, 6)
    assert np.array_equal(closest, oracle.closest_brute("gauss", g, q))
    assert np.array_equal(knn, oracle.knn_brute("gauss", g, q, 6))
    woff, wkeys = ref.radius(q, 9.0)
    for f in (0, capi.QK_WIDE, capi.QK_TUNE_SPLIT, capi.QK_TUNE_LEAF4):
        assert np.array_equal(t.closest(_dev(q), f).cpu().numpy().view(np.uint32), closest), f
        assert np.array_equal(t.knn(_dev(q), 6, f).cpu().numpy().view(np.uint32), knn), f
        off, keys = t.radius(_dev(q), 9.0, f)
        assert np.array_equal(off.cpu().numpy().astype(np.int64), woff), f
        assert np.array_equal(keys.cpu().numpy().view(np.uint64), wkeys), f


@pytest.mark.parametrize("builder", ["sah", "sah4"])
@pytest.mark.parametrize("n", [2, 3, 5, 31, 32, 33, 64, 255, 256, 257, 600, 2048, 2049, 4500, 30011])
@pytest.mark.parametrize("distinct", [1, 9, 1 << 30])
def test_sah_range_edges(cuda, builder, n, distinct):
    """Ranges at the edges of the warp and global tiers, with and without planes that separate the
    centroids: a sound tree, the same one each time, with the oracle's query results."""
    pts = _points(n, n + 1, distinct)
    t = capi.DeviceTree("point", pts, builder=builder)
    assert t.validate() == [0] * 8
    first = t.nodes_bytes().tobytes()
    t.build()
    assert t.nodes_bytes().tobytes() == first
    q = workloads.uniform_points(200, [-5.0] * 3, [105.0] * 3, n, 13)
    ref = oracle.LBVH("point", pts)
    assert np.array_equal(t.knn(_dev(q), 5).cpu().numpy().view(np.uint32), ref.knn(q, 5))


@pytest.mark.parametrize("bins", [4, 17, 32, 33, 64])
def test_sah_bin_counts(cuda, bins):
    tris, _ = workloads.city(700, 11)
    t = capi.DeviceTree("tri", tris, builder="sah", sah_bins=bins)
    assert t.validate() == [0] * 8


@pytest.mark.parametrize("kind", ["tri", "point", "gauss"])
@pytest.mark.parametrize("count", [1, 2, 31, 65, 1000])
def test_few_queries_take_lane_groups(cuda, kind, count):
    """Batches small enough for lane groups, next to schedules that keep one thread per query."""
    items = {"tri": lambda: workloads.terrain(20, 2), "point": lambda: _points(900, 5, 400),
             "gauss": lambda: workloads.gaussians(500, 0.5, 10.0, 4)}[kind]()
    c = items.reshape(len(items), -1)[:, :3]
    q = workloads.uniform_points(count, c.min(0) - 5, c.max(0) + 5, 9, 13)
    t, ref = capi.DeviceTree(kind, items), oracle.LBVH(kind, items)
    r = 0.2 * float(np.linalg.norm(c.max(0) - c.min(0)))  # stashes and chains of every lane
    woff, wkeys = ref.radius(q, r)
    for f in (0, capi.QK_ORDER_MORTON, capi.QK_TUNE_LEAF4):
        assert np.array_equal(t.closest(_dev(q), f).cpu().numpy().view(np.uint32), ref.closest(q)), f
        for k in (3, 8):
            assert np.array_equal(t.knn(_dev(q), k, f).cpu().numpy().view(np.uint32), ref.knn(q, k)), f
        for g in (f, f | capi.QK_TUNE_STASH):
            off, keys = t.radius(_dev(q), r, g)
            assert np.array_equal(off.cpu().numpy().astype(np.int64), woff), g
            assert np.array_equal(keys.cpu().numpy().view(np.uint64), wkeys), g


def test_radius_pool_runs_out_with_lane_groups(cuda):
    """Queries that find nearly every point: the pool holds 128 keys per query, so most are lost and
    traversed again."""
    pts = _points(3000, 6, 1 << 30)
    q = workloads.uniform_points(40, [0.0] * 3, [100.0] * 3, 6, 13)
    t, ref = capi.DeviceTree("point", pts), oracle.LBVH("point", pts)
    off, keys = t.radius(_dev(q), 90.0, capi.QK_TUNE_STASH)
    woff, wkeys = ref.radius(q, 90.0)
    assert np.array_equal(off.cpu().numpy().astype(np.int64), woff)
    assert np.array_equal(keys.cpu().numpy().view(np.uint64), wkeys)


def test_radius_workspace_of_a_large_batch_serves_small_ones(cuda):
    L = capi.lib()
    for flags in (0, capi.QK_TUNE_STASH, capi.QK_TUNE_SPLIT4, capi.QK_WIDE):
        sizes = [L.qk_radius_workspace_bytes(n, flags) for n in (1, 500, 32768, 32769, 40000, 200000)]
        assert sizes == sorted(sizes)


@pytest.mark.parametrize("count", [1, 33, 3552, 3553, 7105, 14208, 14209, 28417, 56833, 113665])
def test_spread_rays(cuda, count):
    """Batches around the sizes where fewer lanes of a warp hold a ray."""
    tris = workloads.terrain(24, 4)
    lo, hi = workloads.bounds_of(tris)
    rays = workloads.down_rays(count, float(lo[0]), float(hi[0]), float(lo[1]), float(hi[1]), 100.0, 4)
    rays[1::3, 3:6] = [0.3, -0.2, -0.9]
    t, ref = capi.DeviceTree("tri", tris), oracle.LBVH("tri", tris)
    t.build_wide()
    want = ref.raycast(rays)
    for f in (0, capi.QK_WIDE, capi.QK_ORDER_COHERENT | capi.QK_TUNE_HIGH_OCC, capi.QK_TUNE_SHORT_STACK,
              capi.QK_TUNE_LEAF4):
        assert np.array_equal(t.raycast(_dev(rays), f).cpu().numpy().view(np.uint64), want), f


@pytest.mark.parametrize("count", [14208, 14209, 28417, 40001, 56833])
def test_spread_queries(cuda, count):
    """Thread-per-query kernels around the sizes where fewer lanes of a warp hold a query."""
    pts = _points(1500, 3, 700)
    q = workloads.uniform_points(count, [-5.0] * 3, [105.0] * 3, 3, 13)
    t, ref = capi.DeviceTree("point", pts), oracle.LBVH("point", pts)
    t.build_wide()
    woff, wkeys = ref.radius(q, 9.0)
    closest, knn = ref.closest(q), ref.knn(q, 9)
    for f in (0, capi.QK_WIDE, capi.QK_TUNE_LEAF4, capi.QK_TUNE_STASH):
        assert np.array_equal(t.closest(_dev(q), f).cpu().numpy().view(np.uint32), closest), f
        assert np.array_equal(t.knn(_dev(q), 9, f).cpu().numpy().view(np.uint32), knn), f
        off, keys = t.radius(_dev(q), 9.0, f)
        assert np.array_equal(off.cpu().numpy().astype(np.int64), woff), f
        assert np.array_equal(keys.cpu().numpy().view(np.uint64), wkeys), f


@pytest.mark.parametrize("flags", [0, capi.QK_ORDER_MORTON, capi.QK_TUNE_SPLIT4, capi.QK_TUNE_SPLIT8,
                                   capi.QK_TUNE_SPLIT, capi.QK_WIDE, capi.QK_TUNE_LEAF4])
@pytest.mark.parametrize("count", [1, 33, 400])
def test_radius_fill_needs_only_the_offsets(cuda, flags, count):
    """Two queries counted before either is filled, in one workspace, and a fill in a workspace of
    its own: without the single-pass flag the fill pass takes nothing but the offsets."""
    import ctypes

    L = capi.lib()
    pts = _points(2000, 4, 900)
    t, ref = capi.DeviceTree("point", pts), oracle.LBVH("point", pts)
    t.build_wide()
    nb = int(L.qk_radius_workspace_bytes(count, flags))
    shared = cuda.zeros(nb, dtype=cuda.uint8, device="cuda")
    jobs = []
    for seed, r in ((1, 12.0), (2, 7.0)):
        q = workloads.uniform_points(count, [-5.0] * 3, [105.0] * 3, seed, 13)
        off = cuda.empty(count + 1, dtype=cuda.int32, device="cuda")
        total = ctypes.c_int64(0)
        head = (ctypes.byref(t.t), _dev(q), count, r, off)
        args = tuple(a.data_ptr() if hasattr(a, "data_ptr") else a for a in head)
        capi.check(L.qk_radius_count(*args, ctypes.byref(total), flags, None, shared.data_ptr(), nb,
                                     None), "qk_radius_count")
        jobs.append((q, r, off, total.value, args, head))
    for q, r, off, total, args, _ in jobs:
        woff, wkeys = ref.radius(q, r)
        assert np.array_equal(off.cpu().numpy().astype(np.int64), woff)
        assert total == len(wkeys)
        for ws in (shared, cuda.zeros(nb, dtype=cuda.uint8, device="cuda")):
            keys = cuda.zeros(max(total, 1), dtype=cuda.int64, device="cuda")
            capi.check(L.qk_radius_fill(*args, keys.data_ptr(), flags, ws.data_ptr(), nb, None),
                       "qk_radius_fill")
            cuda.cuda.synchronize()
            assert np.array_equal(keys.cpu().numpy().view(np.uint64)[:total], wkeys), (flags, r)


@pytest.mark.parametrize("builder", ["sah", "sah4"])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf, 1e25, 3e38])
@pytest.mark.parametrize("n", [40, 256, 257, 700, 9000])
def test_sah_of_coordinates_that_are_not_finite(cuda, builder, bad, n):
    """NaN has no rank and an infinite extent no area: every primitive still gets one slot, every
    node one parent, and the build repeats."""
    pts = workloads.point_cloud("volume", n, 3).copy()
    pts[::5, 0] = bad
    pts[1::11, 2] = -bad
    pts[:2] = bad
    tris = workloads.terrain(int(np.sqrt(n / 2)) + 2, 4).copy()
    tris[::3, 3] = bad
    tris[1::7] = bad
    for kind, items in (("point", pts), ("tri", tris)):
        t = capi.DeviceTree(kind, items, builder=builder)
        m = len(items)
        assert np.array_equal(np.sort(t.host("prim_ids", np.int32)), np.arange(m))
        parent = t.host("parent", np.int32)
        nodes = t.nodes_bytes().view(np.int32).reshape(-1, 8)[: m - 1, 6:]
        assert np.array_equal(np.sort(nodes.reshape(-1)), np.arange(1, 2 * m - 1))
        assert np.array_equal(parent[nodes[:, 0]], np.arange(m - 1))
        assert np.array_equal(parent[nodes[:, 1]], np.arange(m - 1))
        first = t.nodes_bytes().tobytes()
        t.build()
        assert t.nodes_bytes().tobytes() == first


@pytest.mark.parametrize("builder", ["lbvh", "sah"])
@pytest.mark.parametrize("smin,smax", [(0.05, 3.0), (0.01, 30.0)])
def test_few_queries_on_ellipsoids_answer_as_many_do(cuda, builder, smin, smax):
    """Far from the scene a computed distance can be nearer than the boxes around its ellipsoid, so
    results depend on the visit order: a small batch without a schedule flag keeps the order of
    one thread per query."""
    g = workloads.gaussians(700, smin, smax, 5)
    t = capi.DeviceTree("gauss", g, builder=builder)
    rng = np.random.default_rng(7)
    for far in (1e3, 1e6, 1e8):
        q = _dev(rng.uniform(-far, far, (16_000, 3)).astype(np.float32))
        many = cuda.cat([q, q, q])  # 48,000
        for op in (lambda p: t.closest(p), lambda p: t.knn(p, 3), lambda p: t.knn(p, 8)):
            assert cuda.equal(op(q), op(many)[: len(q)]), far


@pytest.mark.parametrize("kind", ["tri", "point"])
@pytest.mark.parametrize("builder", ["lbvh", "sah"])
@pytest.mark.parametrize("n", [2, 3, 4, 5, 9, 700])
def test_few_closest_queries_answer_nan_as_many_do(cuda, kind, builder, n):
    """Queries that are not finite or overflow, and triangles whose first two corners coincide (on
    one side of them the distance is NaN): a batch small enough for lane groups answers each
    query as one thread per query does, which takes the first leaf it meets even when that is NaN."""
    rng = np.random.default_rng(n)
    if kind == "tri":
        items = rng.uniform(0, 10, (n, 9)).astype(np.float32)
        items[::2, 3:6] = items[::2, 0:3]
    else:
        items = rng.uniform(0, 10, (n, 3)).astype(np.float32)
    q = rng.uniform(-15, 25, (700, 3)).astype(np.float32)
    for i, bad in enumerate((np.nan, np.inf, -np.inf, 1e10, 1e19, 3e38)):
        q[i:60:6, i % 3] = bad
    q[60:64] = np.nan
    t = capi.DeviceTree(kind, items, builder=builder)
    many = t.closest(_dev(np.tile(q, (50, 1))))[:len(q)]  # 35,000: one thread per query
    assert cuda.isnan(many[:, 0].contiguous().view(cuda.float32)).any()
    stats = cuda.zeros(4, dtype=cuda.int64, device="cuda")
    assert cuda.equal(t.closest(_dev(q), stats=stats), many)  # counting keeps one thread per query
    for f in (0, capi.QK_ORDER_MORTON, capi.QK_ORDER_COHERENT):
        assert cuda.equal(t.closest(_dev(q), f), many), f
    assert cuda.equal(t.closest(_dev(q[37:38])), many[37:38])


@pytest.mark.parametrize("block,short", [(64, 32), (128, 32), (256, 16), (256, 22), (256, 23), (256, 24)])
def test_batched_queries_with_the_largest_short_stacks(cuda, block, short):
    """Every short stack up to 48 KB per block is taken, beside the kernels' own shared arrays."""
    scenes = [workloads.terrain(k, k) for k in (3, 40, 17)]
    b = capi.Batch("tri", scenes, wide=True)
    b.build()
    b.sync()
    lo, hi = workloads.bounds_of(scenes[1])
    rays = workloads.down_rays(900, float(lo[0]), float(hi[0]), float(lo[1]), float(hi[1]), 100.0, 4)
    pts = workloads.uniform_points(900, lo, hi, 3, 13)
    counts = np.array([300] * 3, np.int32)
    refs = [oracle.LBVH("tri", s) for s in scenes]
    tune = {"block": block, "blocks_per_sm": 2, "short_stack": short, "chunks_per_fetch": 1}
    want = np.concatenate([r.raycast(rays[300 * i:300 * (i + 1)]) for i, r in enumerate(refs)])
    near = np.concatenate([r.closest(pts[300 * i:300 * (i + 1)]) for i, r in enumerate(refs)])
    for flags in (0, capi.QK_WIDE):
        out = cuda.zeros(900, dtype=cuda.int64, device="cuda")
        plan = b.plan(capi.QK_OP_RAY, counts, flags=flags)
        plan.query(_dev(rays), out, tune=tune)
        assert plan.status()[1] == 0
        assert np.array_equal(out.cpu().numpy().view(np.uint64), want), flags
        out = cuda.zeros((900, 2), dtype=cuda.int32, device="cuda")
        plan = b.plan(capi.QK_OP_CLOSEST, counts, flags=flags)
        plan.query(_dev(pts), out, tune=tune)
        assert np.array_equal(out.cpu().numpy().view(np.uint32), near), flags


@pytest.mark.parametrize("kind", ["tri", "point", "gauss"])
@pytest.mark.parametrize("order", [0, capi.QK_ORDER_MORTON])
def test_statistics_are_those_of_one_thread_per_query(cuda, kind, order):
    """Node and leaf counts of a batch small enough for lane groups, against 50 copies of it, which
    is not; the radius results after a counted pass are those of an uncounted one."""
    import ctypes

    L = capi.lib()
    items = {"tri": lambda: workloads.terrain(20, 2), "point": lambda: _points(900, 5, 400),
             "gauss": lambda: workloads.gaussians(500, 0.5, 10.0, 4)}[kind]()
    c = items.reshape(len(items), -1)[:, :3]
    q = workloads.uniform_points(700, c.min(0) - 5, c.max(0) + 5, 9, 13)
    r = 0.15 * float(np.linalg.norm(c.max(0) - c.min(0)))
    t, ref = capi.DeviceTree(kind, items), oracle.LBVH(kind, items)

    def radius(p, flags, stats):
        n = len(p)
        d, off, total = _dev(p), cuda.empty(n + 1, dtype=cuda.int32, device="cuda"), ctypes.c_int64(0)
        nb = int(L.qk_radius_workspace_bytes(n, flags))
        ws = cuda.empty(nb, dtype=cuda.uint8, device="cuda")
        a = (ctypes.byref(t.t), d.data_ptr(), n, r, off.data_ptr())
        capi.check(L.qk_radius_count(*a, ctypes.byref(total), flags, stats.data_ptr(), ws.data_ptr(),
                                     nb, None), "qk_radius_count")
        keys = cuda.zeros(max(total.value, 1), dtype=cuda.int64, device="cuda")
        capi.check(L.qk_radius_fill(*a, keys.data_ptr(), flags, ws.data_ptr(), nb, None),
                   "qk_radius_fill")
        cuda.cuda.synchronize()
        return off.cpu().numpy(), keys.cpu().numpy().view(np.uint64)

    many = np.tile(q, (50, 1))
    ops = [lambda p, s: t.closest(_dev(p), order, stats=s), lambda p, s: t.knn(_dev(p), 4, order, stats=s),
           lambda p, s: radius(p, order, s), lambda p, s: radius(p, order | capi.QK_TUNE_STASH, s)]
    woff, wkeys = ref.radius(q, r)
    for i, op in enumerate(ops):
        few, all50 = (cuda.zeros(4, dtype=cuda.int64, device="cuda") for _ in range(2))
        got = op(q, few)
        op(many, all50)
        assert few[0] > 0 and all50.tolist() == [50 * x for x in few.tolist()], i
        if i >= 2:
            assert np.array_equal(got[0].astype(np.int64), woff)
            assert np.array_equal(got[1], wkeys)


def _closest_wide(wide, wide_ids, items, p):
    """Closest triangle by the 4-wide nodes (child >= 0 a node, < 0 the leaf of slot ~child): near
    children first, equal distances in slot order, the first leaf taken whatever its distance."""
    box = wide.view(np.float32).reshape(-1, 4, 8)
    child = wide.view(np.int32).reshape(-1, 4, 8)[:, :, 6]
    best, best_id, stack, leaves = np.float32(np.inf), -1, [(np.float32(0), 0)], 0
    while stack:
        key, node = stack.pop()
        if best_id >= 0 and not key <= best:
            continue
        hits = []
        for s in range(4):
            if child[node, s] == EMPTY:
                continue
            with np.errstate(invalid="ignore", over="ignore"):
                gap = np.fmax(np.fmax(box[node, s, 0:3] - p, p - box[node, s, 3:6]), np.float32(0))
                d = gap * gap
                d = (d[0] + d[1]) + d[2]
            if best_id < 0 or d <= best:
                hits.append((d, int(child[node, s])))
        hits.sort(key=lambda h: h[0])  # stable
        for d, c in hits:
            if c < 0 and (best_id < 0 or d <= best):
                leaves += 1
                i = int(wide_ids[~c])
                x = np.float32(oracle.prim_dist2("tri", p, items[i]))
                if best_id < 0 or x < best or (x == best and i < best_id):
                    best, best_id = x, i
        stack += [(d, c) for d, c in reversed(hits) if c >= 0 and (best_id < 0 or d <= best)]
    return best, best_id, leaves


EMPTY = -0x80000000


@pytest.mark.parametrize("builder", ["lbvh", "sah"])
def test_wide_children_at_equal_distance_in_slot_order(cuda, builder):
    """Overlapping triangles (queries inside many boxes: equal distances), half of them NaN on one
    side: the answers and the number of leaf tests of a traversal that keeps slot order."""
    rng = np.random.default_rng(5)
    items = rng.uniform(0, 10, (300, 9)).astype(np.float32)
    items[::2, 3:6] = items[::2, 0:3]
    q = rng.uniform(-2, 12, (150, 3)).astype(np.float32)
    t = capi.DeviceTree("tri", items, builder=builder)
    t.build_wide()
    wide = t.host("wide", np.uint8)[: t.t.wide_count * 128]
    ids = t.host("prim_ids", np.int32)
    want = [_closest_wide(wide, ids, items, p) for p in q]
    stats = cuda.zeros(4, dtype=cuda.int64, device="cuda")
    got = t.closest(_dev(q), capi.QK_WIDE, stats=stats).cpu().numpy()
    assert got[:, 1].tolist() == [w[1] for w in want]
    assert np.array_equal(got[:, 0].copy().view(np.float32), np.array([w[0] for w in want]), equal_nan=True)
    assert int(stats[1]) == sum(w[2] for w in want)


@pytest.mark.parametrize("kind", ["tri", "point", "gauss"])
def test_one_thread_per_query_on_request(cuda, kind):
    """QK_TUNE_THREAD: the oracle's results, the counts of a counted call, and the single-pass
    radius in the layout of one chain per query."""
    items = {"tri": lambda: workloads.terrain(20, 2), "point": lambda: _points(900, 5, 400),
             "gauss": lambda: workloads.gaussians(500, 0.5, 10.0, 4)}[kind]()
    c = items.reshape(len(items), -1)[:, :3]
    q = workloads.uniform_points(500, c.min(0) - 5, c.max(0) + 5, 9, 13)
    t, ref = capi.DeviceTree(kind, items), oracle.LBVH(kind, items)
    r = 0.2 * float(np.linalg.norm(c.max(0) - c.min(0)))
    woff, wkeys = ref.radius(q, r)
    th = capi.QK_TUNE_THREAD
    for f in (th, th | capi.QK_ORDER_MORTON, th | capi.QK_ORDER_COHERENT):
        assert np.array_equal(t.closest(_dev(q), f).cpu().numpy().view(np.uint32), ref.closest(q)), f
        for k in (3, 8, 16):
            assert np.array_equal(t.knn(_dev(q), k, f).cpu().numpy().view(np.uint32), ref.knn(q, k)), f
        for g in (f, f | capi.QK_TUNE_STASH):
            off, keys = t.radius(_dev(q), r, g)
            assert np.array_equal(off.cpu().numpy().astype(np.int64), woff), g
            assert np.array_equal(keys.cpu().numpy().view(np.uint64), wkeys), g
    size = capi.lib().qk_radius_workspace_bytes
    assert size(500, capi.QK_TUNE_STASH | th) < size(500, capi.QK_TUNE_STASH)
    a, b = (cuda.zeros(4, dtype=cuda.int64, device="cuda") for _ in range(2))
    t.closest(_dev(q), th, stats=a)
    t.closest(_dev(q), 0, stats=b)
    assert cuda.equal(a, b)


@pytest.mark.parametrize("n", [4097, 8192, 12289, 70001])
@pytest.mark.parametrize("bits", [8, 16, 24, 32])
@pytest.mark.parametrize("spread", [1, 3, 1 << 32])
@pytest.mark.parametrize("max_polls,wide_states", [(-1, 0), (0, 0), (-1, 1), (4096, 1)])
def test_sort_paths_few_calls_take(cuda, n, bits, spread, max_polls, wide_states):
    """Tiles that count the earlier keys themselves (every one, or those whose first read is empty)
    and 64-bit tile states, after an even and an odd number of passes."""
    L = capi.lib()
    rng = np.random.default_rng(n + bits)
    keys = (rng.integers(0, spread, n, dtype=np.uint64) & ((1 << bits) - 1)).astype(np.uint32)
    vals = rng.integers(0, 1 << 32, n, dtype=np.uint64).astype(np.uint32)
    kin, vin = (_dev(a.view(np.int32), np.int32) for a in (keys, vals))
    kout, vout = cuda.empty_like(kin), cuda.empty_like(vin)
    nb = int(L.qk_sort_workspace_bytes_paths(n, wide_states))
    assert nb >= int(L.qk_sort_workspace_bytes(n))
    ws = cuda.empty(nb, dtype=cuda.uint8, device="cuda")
    capi.check(L.qk_sort_pairs_paths(kin.data_ptr(), vin.data_ptr(), kout.data_ptr(), vout.data_ptr(), n,
                                     bits, max_polls, wide_states, ws.data_ptr(), nb, None),
               "qk_sort_pairs_paths")
    cuda.cuda.synchronize()
    o = np.argsort(keys, kind="stable")
    assert np.array_equal(kout.cpu().numpy().view(np.uint32), keys[o])
    assert np.array_equal(vout.cpu().numpy().view(np.uint32), vals[o])
