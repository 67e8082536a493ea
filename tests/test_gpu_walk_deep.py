"""Deep chains of wide node groups (imported Node1 trees): at every level one
node of a group goes on, so the reference's own stack holds one range however
deep the chain is, and the warp's pool of node ranges must not need more than
it has.  Against the oracle, and box-test totals counted from the tree."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def chain(oracle, depth, group, at, side_boxes=None):
    """`depth` groups of `group` nodes: node `at` of a group is the next
    level's parent (its box holds every ray), the others are leaves with
    side_boxes[j] (by default where no ray goes)."""
    far = ((1e6, 1e6, 1e6), (1e6 + 1, 1e6 + 1, 1e6 + 1))
    tris = np.array([[-50, -50, 1.5, 50, -50, 1.5, 0, 50, 1.5]], np.float32)
    nodes = np.zeros(1 + depth * group, oracle.NODE1)
    big = ((-100, -100, 1), (100, 100, 20))
    nodes[0] = (big[0], group, 0, big[1], 1)
    for d in range(depth):
        for j in range(group):
            i = 1 + d * group + j
            lo, hi = side_boxes[j] if side_boxes else far
            nodes[i] = (lo, 1, 1, hi, 0)
            if j == at:
                last = d == depth - 1
                nodes[i] = (big[0], 1 if last else group, 1 if last else 0, big[1], 0 if last else 1 + (d + 1) * group)
    return nodes, tris


@pytest.mark.parametrize("group,at", [(2, 0), (16, 0), (16, 15), (17, 16), (40, 3), (40, 39), (200, 199)])
@pytest.mark.parametrize("rays", [1, 32, 97])
def test_reference_rays(ctx, oracle, group, at, rays):
    nodes, tris = chain(oracle, 300, group, at)
    bvh = ctx.import_node1(nodes, 0, tris)
    r = np.zeros((rays, 8), np.float32)
    r[:, 0] = np.linspace(-60, 60, rays)
    r[:, 6], r[:, 7] = 1.0, 10000.0
    r[:, 4:6] = 1e-3
    ids, _, tests = oracle.trace(nodes, 0, tris, r, 0)
    assert (tests == 1 + 300 * group).all()
    for got in (ctx.trace(bvh, "ref", rays=r)[0], ctx.traverse(bvh, 0, 1, r)):
        assert np.array_equal(got["id"], ids) and np.array_equal(got["tests"], tests)
    assert ctx.sync() == 0
    bvh.free()


@pytest.mark.parametrize("k,w,h", [(1, 4, 2), (2, 3, 4), (4, 6, 4), (8, 6, 8)])
@pytest.mark.parametrize("group,at", [(2, 0), (17, 16), (40, 39)])
def test_packets(ctx, oracle, k, w, h, group, at):
    depth = 400
    nodes, tris = chain(oracle, depth, group, at)
    bvh = ctx.import_node1(nodes, 0, tris)
    _, heat = ctx.trace(bvh, "packet", k=k, camera="reference", width=w, height=h, origin=(0, 0, 0))
    assert ctx.trace_stats()["box_tests"] == w * h // k * (1 + depth * group)
    assert np.array_equal(heat, oracle.trace_coherent(nodes, 0, w, h, (0, 0, 0), False, k))
    assert ctx.sync() == 0
    bvh.free()


# four tiles, each with `fans` leaf boxes a group that only some of its packets'
# directions can hit: the packets go on alone there, each to test that one box
@pytest.mark.parametrize("k,side", [(16, 4), (64, 8)])
@pytest.mark.parametrize("fans,at", [(1, 4), (9, 0), (39, 156), (39, 60)])
def test_bundles(ctx, oracle, k, side, fans, at):
    depth = 60
    group = 4 * fans + 1
    boxes = []
    for j in range(group):
        q = (j if j < at else j - 1) % 4
        x, y = (8.0 if q & 1 else -8.0), (8.0 if q & 2 else -8.0)
        boxes.append(((x - 0.1, y - 0.1, 10.0), (x + 0.1, y + 0.1, 10.1)))
    nodes, tris = chain(oracle, depth, group, at, boxes)
    bvh = ctx.import_node1(nodes, 0, tris)
    n = 2 * side
    _, heat = ctx.trace(bvh, "bundle", k=k, camera="reference", width=n, height=n, origin=(0, 0, 0))
    packets = k // 8
    assert ctx.trace_stats()["box_tests"] == 4 * (1 + depth * group) + 4 * packets * depth * fans
    assert np.array_equal(heat, oracle.trace_coherent(nodes, 0, n, n, (0, 0, 0), True, k))
    assert ctx.sync() == 0
    bvh.free()
