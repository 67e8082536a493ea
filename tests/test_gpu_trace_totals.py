"""Trace statistics of the 8-wide refill kernels, whose lanes keep 32-bit
totals and hand them on before they are full (here: long before): the same
sums as kept to the end, and the box tests of the hits."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["closest", "anyhit"])
@pytest.mark.parametrize("heatmap", [False, True])
def test_totals_handed_on(lib_built, mode, heatmap):
    import sequoia_gb300 as sq
    from sequoia_gb300 import scenes
    ctx = sq.Context(0)
    tris = scenes.gaussian_soup(20_000, 3, seed=71)
    lo, hi = scenes.scene_box(tris)
    rays = scenes.random_rays(400_000, lo, hi, seed=72)
    bvh = ctx.build(tris, "morton", wide=True)
    cam = dict(camera="pinhole", width=200, height=100, origin=(0, 0, -40), target=(0, 0, 0), vfov=40.0)
    calls = [lambda: ctx.trace(bvh, mode, rays=rays, heatmap=heatmap),
             lambda: ctx.trace(bvh, mode, sched="refill", heatmap=heatmap, **cam),
             lambda: ctx.trace_batches(bvh, mode, [rays[:100_001], cam, rays[100_001:]], heatmap=heatmap)]
    for call in calls:
        hits, _ = call()
        want = ctx.trace_stats()
        assert want["box_tests"] == hits["tests"].sum(dtype=np.uint64)
        ctx.debug_inject("force", ctx.FORCE_SMALL_TOTALS)
        again, _ = call()
        got = ctx.trace_stats()
        ctx.debug_inject("off")
        assert np.array_equal(again["tests"], hits["tests"])
        # (which of two any-hit candidates a ray meets first does not depend on its lane)
        assert got == want
    ctx.close()
