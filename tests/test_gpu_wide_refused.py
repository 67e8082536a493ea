"""8-wide trees whose collapse refuses a node (a leaf of more than 15
triangles, a root record of more than eight): the error is reported once, and
the tree holds an empty node there whatever the recycled device memory held
before, so that a trace of it is safe and finds the rest."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ERR_DEVICE = 4
NODE_COUNT = 0x10
NONE = 0xFFFFFFFF


def raw_sync(ctx):
    import sequoia_gb300 as sq
    bits = C.c_uint32()
    st = sq.load_library().sq_sync(ctx.handle, C.byref(bits))
    return st, bits.value


def fill_cache(ctx, word):
    """Blocks of many sizes full of `word` in the context's allocator."""
    n = 16
    while n < 400_000:
        keys = np.full(n, word, np.uint32)
        ctx.radix_sort_pairs(keys, keys)
        n = n * 3 // 2


def shapes():
    from sequoia_gb300 import scenes
    soup = scenes.gaussian_soup(3000, 2, seed=31)
    same = soup.copy()
    same[1000:1200] = soup[7]  # one leaf of 200
    return {"leaves": (soup, 40), "same": (same, 8), "root9": (np.repeat(soup[:1], 9, 0), 8),
            "root16": (np.repeat(soup[:1], 16, 0), 8)}


@pytest.mark.parametrize("builder", ["sah", "grid"])
@pytest.mark.parametrize("shape", ["leaves", "same", "root9", "root16"])
@pytest.mark.parametrize("word", [NONE, 0x7FFFFFFF])
def test_refused_build(lib_built, builder, shape, word):
    import sequoia_gb300 as sq
    import torch
    from sequoia_gb300 import scenes
    ctx = sq.Context(0)
    tris, leaf = shapes()[shape]
    lo, hi = scenes.scene_box(tris)
    rays = scenes.random_rays(3000, lo, hi, seed=5)
    fill_cache(ctx, word)
    bvh = ctx.build(tris, builder, leaf=leaf, wide=True)
    out = torch.zeros(3 * len(rays), dtype=torch.int32, device="cuda")
    ctx.trace(bvh, "closest", rays=rays, hits=out)  # before the error is asked for
    st, bits = raw_sync(ctx)
    # (nine triangles with one centroid are a leaf child of a grid's tree)
    refused = not (builder == "grid" and shape == "root9")
    assert (st, bits) == ((ERR_DEVICE, NODE_COUNT) if refused else (0, 0))
    got = out.cpu().numpy().view(np.uint32).reshape(-1, 3)
    whole = ctx.build(tris, "morton")  # (a cluster of more than eight overflows the binary traversal's hit list)
    want, _ = ctx.trace(whole, "closest", rays=rays)
    for sched in ("tiles", "refill"):
        again, _ = ctx.trace(bvh, "closest", rays=rays, sched=sched)
        assert np.array_equal(again["id"], got[:, 0]) and np.array_equal(again["tests"], got[:, 2])
        hit = again["id"] != NONE
        assert (again["id"][hit] < len(tris)).all() and (want["id"][hit] != NONE).all()
        assert (again["t"][hit] >= want["t"][hit]).all()
        if refused and shape.startswith("root"):
            assert not hit.any()
        assert shape != "same" or hit.any()
    assert raw_sync(ctx) == (0, 0)
    bvh.free()
    whole.free()
    ctx.close()


def test_refused_batch(lib_built):
    import sequoia_gb300 as sq
    from sequoia_gb300 import scenes
    from test_gpu_batch import separate
    ctx = sq.Context(0)
    soup = scenes.gaussian_soup(3000, 2, seed=31)
    lo, hi = scenes.scene_box(soup)
    rays = scenes.random_rays(500, lo, hi, seed=6)
    good = [dict(tris=soup, rays=rays), dict(tris=soup[:9], rays=rays)]
    fill_cache(ctx, NONE)
    for graph in (False, True):
        with pytest.raises(sq.SequoiaError) as e:
            ctx.batch([good[0], dict(tris=np.repeat(soup[:1], 16, 0), rays=rays), good[1]], builder="sah", wide=True,
                      graph=graph)
        assert e.value.status == ERR_DEVICE and "0x10 " in str(e.value)
        assert raw_sync(ctx) == (0, 0)
    want = separate(ctx, good, "closest", True, "sah")
    b = ctx.batch(good, builder="sah", wide=True)
    got, _ = b.run()
    assert np.array_equal(got["id"], want["id"]) and np.array_equal(got["t"], want["t"])
    b.free()
    ctx.close()


@pytest.mark.parametrize("builder", ["sah", "grid"])
@pytest.mark.parametrize("wide", [False, True])
def test_range_past_the_record_count(lib_built, builder, wide):
    """A leaf range of more than 65535 triangles, which no record can hold."""
    import sequoia_gb300 as sq
    from sequoia_gb300 import scenes
    ctx = sq.Context(0)
    soup = scenes.gaussian_soup(500, 2, seed=33)
    lo, hi = scenes.scene_box(soup)
    rays = scenes.random_rays(2000, lo, hi, seed=8)
    far = soup[:1] + np.float32(1000)
    alone = ctx.build(soup, builder, wide=wide)
    want, _ = ctx.trace(alone, "closest", rays=rays)
    for tris in (np.concatenate([soup, np.repeat(far, 70_000, 0)]), np.repeat(far, 70_000, 0)):
        fill_cache(ctx, NONE)
        bvh = ctx.build(np.ascontiguousarray(tris), builder, wide=wide)
        assert raw_sync(ctx) == (ERR_DEVICE, NODE_COUNT)
        for sched in ("tiles", "refill"):
            got, _ = ctx.trace(bvh, "closest", rays=rays, sched=sched)
            if len(tris) > 70_000:
                assert np.array_equal(got["id"], want["id"]) and np.array_equal(got["t"], want["t"])
            else:
                assert (got["id"] == NONE).all()
        ref, _ = ctx.trace(bvh, "ref", rays=rays)
        assert len(tris) > 70_000 or (ref["id"] == NONE).all()
        assert raw_sync(ctx) == (0, 0)
        bvh.free()
    alone.free()
    ctx.close()


def test_collapse_that_gave_up_is_an_empty_tree(lib_built):
    import sequoia_gb300 as sq
    import torch
    from sequoia_gb300 import scenes
    ctx = sq.Context(0)
    tris = scenes.gaussian_soup(20_000, 4, seed=35)
    lo, hi = scenes.scene_box(tris)
    rays = scenes.random_rays(3000, lo, hi, seed=9)
    for word in (NONE, 0x7FFFFFFF):
        fill_cache(ctx, word)
        ctx.debug_inject("stall_barrier", 256)
        bvh = ctx.build(tris, "morton", wide=True)
        out = torch.ones(3 * len(rays), dtype=torch.int32, device="cuda")
        ctx.trace(bvh, "closest", rays=rays, hits=out)
        st, bits = raw_sync(ctx)
        assert st == ERR_DEVICE and bits == 0x8
        got = out.cpu().numpy().view(np.uint32).reshape(-1, 3)
        assert (got[:, 0] == NONE).all() and (got[:, 2] == 0).all()
        info = bvh.info()
        assert (info.wide_nodes, info.wide_levels) == (1, 1)
        bvh.free()
    ctx.close()
