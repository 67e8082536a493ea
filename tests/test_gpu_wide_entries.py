"""The binary refill kernels with 16-byte stack entries, which trees of more
than 2^27 records take: the same hits, distances and box tests as with the
8-byte entries and as the tiles schedule, on trees of the usual sizes."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture
def wctx(lib_built):
    import sequoia_gb300 as sq
    ctx = sq.Context(0)
    ctx.debug_inject("force", ctx.FORCE_WIDE_ENTRIES)
    yield ctx
    ctx.close()


def compare(ctx, bvh, mode, rays):
    got = [ctx.trace(bvh, mode, rays=rays, binary=True, sched="refill")[0],
           ctx.trace_batches(bvh, mode, [rays[:37], rays[37:]], binary=True)[0]]
    want = ctx.trace(bvh, mode, rays=rays, binary=True, sched="tiles")[0]
    for g in got:
        assert np.array_equal(g["tests"], want["tests"])
        assert np.array_equal(g["id"], want["id"]) and np.array_equal(g["t"], want["t"])
    assert ctx.sync() == 0


@pytest.mark.parametrize("builder,leaf", [("morton", 8), ("sah", 1), ("sah", 8), ("grid", 4)])
@pytest.mark.parametrize("mode", ["closest", "anyhit"])
def test_builds(wctx, builder, leaf, mode):
    from sequoia_gb300 import scenes
    tris = scenes.gaussian_soup(30_000, 3, seed=51)
    rays = scenes.random_rays(5000, *scenes.scene_box(tris), seed=52)
    compare(wctx, wctx.build(tris, builder, leaf=leaf), mode, rays)


# leaves of any count and groups of three to eight nodes
@pytest.mark.parametrize("big", [1, 15, 16, 400])
@pytest.mark.parametrize("fan", [3, 8])
@pytest.mark.parametrize("mode", ["closest", "anyhit"])
def test_imported(wctx, oracle, big, fan, mode):
    from sequoia_gb300 import scenes
    tris = scenes.gaussian_soup(big * fan * fan, 1, seed=big)
    nodes = np.zeros(1 + fan + fan * fan, oracle.NODE1)

    def put(i, lo, hi, child, count, leaf):
        v = tris[lo:hi].reshape(-1, 3)
        nodes[i] = (v.min(0), count, leaf, v.max(0), child)

    put(0, 0, len(tris), 1, fan, 0)
    for j in range(fan):
        put(1 + j, j * fan * big, (j + 1) * fan * big, 1 + fan + j * fan, fan, 0)
        for q in range(fan):
            first = (j * fan + q) * big
            put(1 + fan + j * fan + q, first, first + big, first, big, 1)
    rays = scenes.random_rays(1000, *scenes.scene_box(tris), seed=7)
    compare(wctx, wctx.import_node1(nodes, 0, tris), mode, rays)


@pytest.mark.parametrize("mode", ["closest", "anyhit"])
def test_mesh_batch(wctx, mode):
    from sequoia_gb300 import scenes
    meshes = []
    for j, n in enumerate((700, 3, 9000)):
        tris = scenes.gaussian_soup(n, 1, seed=60 + j)
        meshes.append(dict(tris=tris, rays=scenes.random_rays(300 + j, *scenes.scene_box(tris), seed=j)))
    b = wctx.batch(meshes, mode=mode, wide=False)
    got, _ = b.run()
    wctx.debug_inject("off")
    narrow = wctx.batch(meshes, mode=mode, wide=False)
    want, _ = narrow.run()
    for key in ("id", "t", "tests"):
        assert np.array_equal(got[key], want[key]), key


def test_child_index_past_the_records(wctx, oracle):
    import sequoia_gb300 as sq
    from test_gpu_bad_records import tree
    for child in (1 << 27, 0x87FFFFFF, 0xFFFFFFFE):
        nodes, tris = tree(oracle, child, 2)
        bvh = wctx.import_node1(nodes, 0, tris)
        rays = np.zeros((40, 8), np.float32)
        rays[:, 0:2], rays[:, 6], rays[:, 7] = 0.9, 1.0, 100.0
        with pytest.raises(sq.SequoiaError):
            wctx.trace(bvh, "closest", rays=rays, sched="refill")
        bits = C.c_uint32()
        assert sq.load_library().sq_sync(wctx.handle, C.byref(bits)) == 0
