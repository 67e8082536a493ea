"""Packet images on both sides of the size from which a warp takes a share of
the packets left instead of four, with counts that no share divides: the
oracle's heatmap bytes, and the box tests of all packets once."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 100, 5000, 140_000])
@pytest.mark.parametrize("k,sizes", [(1, [(128, 128), (331, 257)]), (2, [(331, 514)]), (4, [(334, 1002)]),
                                     (8, [(90, 1004), (670, 1004)])])
def test_packet_images(ctx, oracle, n, k, sizes):
    from sequoia_gb300 import scenes
    tris = scenes.gaussian_soup(n, 1 + n // 20_000, seed=n)
    lo, hi = scenes.scene_box(tris)
    c = (lo + hi) * np.float32(0.5)
    origin = np.array([c[0], c[1], lo[2] - np.float32(0.5) * (hi[2] - lo[2])], np.float32)
    bvh = ctx.build(tris, "sah")
    nodes, root = bvh.export_node1()
    for w, h in sizes:
        _, heat = ctx.trace(bvh, "packet", k=k, camera="reference", width=w, height=h, origin=origin)
        assert np.array_equal(heat, oracle.trace_coherent(nodes, root, w, h, origin, False, k))
        first = ctx.trace_stats()["box_tests"]
        assert first >= w * h // k
        ctx.trace(bvh, "packet", k=k, camera="reference", width=w, height=h, origin=origin)
        assert ctx.trace_stats()["box_tests"] == first
    assert ctx.sync() == 0
    bvh.free()
