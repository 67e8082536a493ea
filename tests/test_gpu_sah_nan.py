"""SAH and grid builds of meshes with NaN and infinite vertices: a NaN bound is
passed over, as in the reference's min and max, in every phase of the builder.
Record for record the oracle's trees, and batches the same as separate builds."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NAN, NEG_NAN = (np.array([u], np.uint32).view(np.float32)[0] for u in (0x7FC00000, 0xFFC00001))


def spoiled(n, kind, seed):
    from sequoia_gb300 import scenes
    rng = np.random.default_rng(seed)
    tris = scenes.gaussian_soup(n, 1 + n // 3000, seed=seed)
    some = rng.integers(0, n, max(1, n // 40))
    tris[some, rng.integers(0, 9, len(some))] = {"nan": NAN, "-nan": NEG_NAN}.get(kind, np.inf)
    if kind == "mixed":
        some = rng.integers(0, n, max(1, n // 40))
        tris[some, rng.integers(0, 9, len(some))] = np.where(rng.integers(0, 2, len(some)), NAN, -np.inf)
    if kind == "axis":
        tris[rng.permutation(n)[: n // 2], 0::3] = NAN  # no bound at all on x
    return tris


def records(nodes, root):
    """Every reachable record in order, NaNs alike."""
    out, todo = [], [int(root)]
    while todo:
        r = nodes[todo.pop()]
        box = np.array([*r["min"], *r["max"]], np.float32)
        box[np.isnan(box)] = NAN
        out.append((box.tobytes(), int(r["count"]), int(r["flags"]), int(r["child"])))
        if not r["flags"] & 1:
            todo.extend(range(int(r["child"]), int(r["child"]) + int(r["count"])))
    return out


# one size for each phase of the builder: warp, block, chunks of 256, and the
# grid's cells of any of them
@pytest.mark.parametrize("n", [1, 6, 130, 1100, 20_000])
@pytest.mark.parametrize("kind", ["nan", "-nan", "inf", "mixed", "axis"])
@pytest.mark.parametrize("bins", [3, 8, 9, 16, 32])
def test_trees(ctx, oracle, n, kind, bins):
    tris = spoiled(n, kind, 100 * n + bins)
    for builder in ("sah", "grid"):
        bvh = ctx.build(tris, builder, bins=bins, leaf=4)
        want = (oracle.build_sah if builder == "sah" else oracle.build_grid)(tris, bins, 4)
        assert records(*bvh.export_node1()) == records(*want[:2]), builder
        bvh.free()
    assert ctx.sync() == 0


@pytest.mark.parametrize("kind", ["nan", "mixed", "axis"])
@pytest.mark.parametrize("bins", [8, 16, 32])
def test_batch(ctx, kind, bins):
    from sequoia_gb300 import scenes
    from test_gpu_batch import separate
    meshes = [dict(tris=spoiled(n, kind, n + bins), rays=scenes.random_rays(400, np.float32([-12] * 3),
                                                                            np.float32([12] * 3), seed=n))
              for n in (1, 6, 130, 1100, 3000)]
    want = separate(ctx, meshes, "ref", False, "sah", bins=bins, leaf=4)
    b = ctx.batch(meshes, mode="ref", wide=False, builder="sah", bins=bins, leaf=4)
    got, _ = b.run()
    assert np.array_equal(got["id"], want["id"]) and np.array_equal(got["tests"], want["tests"])
    assert ctx.sync() == 0
    b.free()
