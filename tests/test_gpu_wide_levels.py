"""The 8-wide collapse as one launch per level, the path of a device without
cooperative launches: the same trees as the cooperative kernel's (node and
level counts, hits, distances, box tests), in single builds and batches."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def lctx(lib_built):
    import sequoia_gb300 as sq
    ctx = sq.Context(0)
    yield ctx
    ctx.close()


def same_trees(ctx, a, b, rays):
    ia, ib = a.info(), b.info()
    assert (ia.wide_nodes, ia.wide_levels) == (ib.wide_nodes, ib.wide_levels)
    for mode in ("closest", "anyhit"):
        for sched in ("tiles", "refill"):
            ga, gb = (ctx.trace(t, mode, rays=rays, sched=sched)[0] for t in (a, b))
            assert np.array_equal(ga["id"] != 0xFFFFFFFF, gb["id"] != 0xFFFFFFFF)
            assert np.array_equal(ga["tests"], gb["tests"])
            if mode == "closest":
                assert np.array_equal(ga["id"], gb["id"]) and np.array_equal(ga["t"], gb["t"])


# a root alone, a root of clusters, more tasks than a block, more levels than
# the four task counters that take turns
@pytest.mark.parametrize("n", [0, 1, 2, 9, 70, 1000, 60_000])
@pytest.mark.parametrize("builder", ["morton", "sah", "grid"])
def test_single_build(lctx, builder, n):
    from sequoia_gb300 import scenes
    tris = scenes.gaussian_soup(n, 3, seed=41 + n) if n else np.zeros((0, 9), np.float32)
    lo, hi = scenes.scene_box(tris) if n else (np.zeros(3, np.float32), np.ones(3, np.float32))
    rays = scenes.random_rays(700, lo, hi, seed=n)
    coop = lctx.build(tris, builder, wide=True)
    lctx.debug_inject("force", lctx.FORCE_LEVEL_COLLAPSE)
    level = lctx.build(tris, builder, wide=True)
    lctx.debug_inject("off")
    if n == 60_000:
        assert level.info().wide_levels > 4
    assert level.info().wide_launches != coop.info().wide_launches
    same_trees(lctx, coop, level, rays)
    assert lctx.sync() == 0


def test_unknown_path_is_refused(lctx):
    import sequoia_gb300 as sq
    with pytest.raises(sq.SequoiaError) as e:
        lctx.debug_inject("force", 1 << 30)
    assert e.value.status == 1


@pytest.mark.parametrize("builder", ["morton", "sah"])
@pytest.mark.parametrize("graph", [False, True])
def test_batch(lctx, builder, graph):
    from sequoia_gb300 import scenes
    from test_gpu_batch import separate
    meshes = []
    for j, n in enumerate([0, 1, 7, 40_000, 300, 0, 2500] + list(range(1, 30))):
        tris = scenes.gaussian_soup(n, 1, seed=600 + j) if n else np.zeros((0, 9), np.float32)
        lo, hi = scenes.scene_box(tris) if n else (np.zeros(3, np.float32), np.ones(3, np.float32))
        meshes.append(dict(tris=tris, rays=scenes.random_rays(60 + j, lo, hi, seed=j)))
    want = separate(lctx, meshes, "closest", True, builder)
    lctx.debug_inject("force", lctx.FORCE_LEVEL_COLLAPSE)
    b = lctx.batch(meshes, mode="closest", wide=True, builder=builder, graph=graph)
    for _ in range(2):
        got, _ = b.run()
        for key in ("id", "t", "tests"):
            assert np.array_equal(got[key], want[key]), key
    lctx.debug_inject("off")
    assert lctx.sync() == 0
    b.free()
