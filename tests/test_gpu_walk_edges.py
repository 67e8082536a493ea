"""Traversal at the edges of its splits: a warp's shared pool of node ranges
(reference tracer, packets, bundles), stack entries that hold a child's own
range (binary refill), and batches whose meshes end at tile edges.  Against
the oracle or a mesh's own build: the same bytes and counts."""
import numpy as np
import pytest

from test_gpu_batch import separate

pytestmark = pytest.mark.gpu


def overlapping(n, seed=3):
    """n large triangles through one point: a ray enters nearly every node."""
    rng = np.random.default_rng(seed)
    d = rng.normal(size=(n, 3, 3)).astype(np.float32)
    d -= d.mean(1, keepdims=True)
    return (d * np.float32(4.0)).reshape(n, 9)


def camera_of(tris):
    v = tris.reshape(-1, 3)
    lo, hi = v.min(0), v.max(0)
    c = (lo + hi) * np.float32(0.5)
    return np.array([c[0], c[1], np.float32(2) * lo[2] - c[2]], np.float32)


# one owner, a full and a ragged group of owners; trees of one node, of a pool
# that never fills and of one that does (a node range per owner and box)
@pytest.mark.parametrize("n", [1, 40, 3000])
@pytest.mark.parametrize("builder", ["morton", "sah", "grid"])
@pytest.mark.parametrize("mode,k,sizes", [("packet", 1, [(1, 1), (5, 3)]), ("packet", 2, [(1, 2), (9, 6)]),
                                          ("packet", 4, [(2, 2), (10, 6)]), ("packet", 8, [(2, 4), (10, 12)]),
                                          ("bundle", 16, [(4, 4), (12, 4), (20, 12)]),
                                          ("bundle", 64, [(8, 8), (24, 8)])])
def test_pool_of_packets_and_bundles(ctx, oracle, n, builder, mode, k, sizes):
    tris = overlapping(n)
    bvh = ctx.build(tris, builder)
    nodes, root = bvh.export_node1()
    for origin in (camera_of(tris), np.array([0.1, 0.2, 0.3], np.float32)):  # outside, and among the triangles
        for w, h in sizes:
            _, heat = ctx.trace(bvh, mode, k=k, camera="reference", width=w, height=h, origin=origin)
            assert np.array_equal(heat, oracle.trace_coherent(nodes, root, w, h, origin, mode == "bundle", k)), (w, h)
    assert ctx.sync() == 0
    bvh.free()


@pytest.mark.parametrize("n", [1, 40, 3000])
@pytest.mark.parametrize("builder", ["morton", "sah", "grid"])
@pytest.mark.parametrize("rays", [1, 31, 33, 97])
def test_pool_of_rays(ctx, oracle, n, builder, rays):
    from sequoia_gb300 import scenes
    tris = overlapping(n, seed=n)
    r = scenes.random_rays(rays, np.float32([-3, -3, -3]), np.float32([3, 3, 3]), seed=rays)
    bvh = ctx.build(tris, builder)
    nodes, root = bvh.export_node1()
    ids, _, tests = oracle.trace(nodes, root, tris, r, 0)
    hits, _ = ctx.trace(bvh, "ref", rays=r)
    assert np.array_equal(hits["id"], ids) and np.array_equal(hits["tests"], tests)
    assert ctx.sync() == 0
    bvh.free()


# leaves of 15 triangles fit a stack entry, of 16 and more do not
@pytest.mark.parametrize("big", [1, 15, 16, 40])
@pytest.mark.parametrize("mode", ["closest", "anyhit"])
def test_refill_entries_of_large_leaves(ctx, oracle, big, mode):
    from sequoia_gb300 import scenes
    leaves = [big, 15, 3, 16]
    tris = scenes.gaussian_soup(sum(leaves), 1, seed=big)
    nodes = np.zeros(7, oracle.NODE1)
    first = np.cumsum([0] + leaves)

    def put(i, lo, hi, child, count, leaf):
        v = tris[lo:hi].reshape(-1, 3)
        nodes[i] = (v.min(0), count, 1 if leaf else 0, v.max(0), child)

    put(0, 0, first[4], 1, 2, False)
    put(1, 0, first[2], 3, 2, False)
    put(2, first[2], first[4], 5, 2, False)
    for j in range(4):
        put(3 + j, first[j], first[j + 1], first[j], leaves[j], True)
    bvh = ctx.import_node1(nodes, 0, tris)
    v = tris.reshape(-1, 3)
    rays = scenes.random_rays(1000, v.min(0), v.max(0), seed=7)
    ids, ts, tests = oracle.trace(nodes, 0, tris, rays, 1 if mode == "closest" else 2)
    for sched in ("refill", "tiles"):
        hits, _ = ctx.trace(bvh, mode, rays=rays, binary=True, sched=sched)
        assert np.array_equal(hits["tests"], tests), sched
        if mode == "closest":
            assert np.array_equal(hits["id"], ids) and np.array_equal(hits["t"], ts), sched
        else:
            assert np.array_equal(hits["id"] != 0xFFFFFFFF, ids != 0xFFFFFFFF), sched
    assert ctx.sync() == 0
    bvh.free()


# meshes that begin and end inside, at and beside the edges of 256-triangle
# tiles, and many trees in one collapse
@pytest.mark.parametrize("builder", ["morton", "sah"])
@pytest.mark.parametrize("wide", [False, True])
def test_batch_mesh_edges(ctx, builder, wide):
    from sequoia_gb300 import scenes
    sizes = [255, 1, 0, 256, 257, 2, 511, 0, 0, 1, 513, 9, 1024, 3, 129, 128] + list(range(1, 41)) + [2048, 7]
    meshes = []
    for j, n in enumerate(sizes):
        tris = scenes.gaussian_soup(n, 1, seed=500 + j) if n else np.zeros((0, 9), np.float32)
        lo, hi = (tris.reshape(-1, 3).min(0), tris.reshape(-1, 3).max(0)) if n else (np.zeros(3), np.ones(3))
        meshes.append(dict(tris=tris, rays=scenes.random_rays(50 + j, lo, hi, seed=j)))
    want = separate(ctx, meshes, "closest", wide, builder)
    b = ctx.batch(meshes, mode="closest", wide=wide, builder=builder)
    for _ in range(2):
        got, _ = b.run()
        for key in ("id", "t", "tests"):
            assert np.array_equal(got[key], want[key]), key
    assert ctx.sync() == 0
    b.free()


@pytest.mark.parametrize("block", [64, 128, 256])
def test_batch_reference_tracer_blocks(ctx, block):
    from sequoia_gb300 import scenes
    meshes = []
    for j, n in enumerate((700, 3, 2000)):
        tris = overlapping(n, seed=j)
        meshes.append(dict(tris=tris, rays=scenes.random_rays(33 + 40 * j, np.float32([-3] * 3), np.float32([3] * 3),
                                                              seed=j)))
    want = separate(ctx, meshes, "ref", False)
    b = ctx.batch(meshes, mode="ref", wide=False, block=block)
    got, _ = b.run()
    assert np.array_equal(got["tests"], want["tests"])
    assert np.array_equal(got["id"] != 0xFFFFFFFF, want["id"] != 0xFFFFFFFF)
    assert ctx.sync() == 0
    b.free()
