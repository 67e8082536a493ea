"""SAH builds at the edges of the builder's phases (subtrees of a warp up to
128 triangles, of a block up to 1024, levels of chunks beyond) and of its bin
groupings (up to 8, 16 and 32 bins), against the oracle: the same records, so
every comparison is exact."""
import numpy as np
import pytest

from test_gpu_lbvh import assert_same_tree

pytestmark = pytest.mark.gpu

SIZES = [2, 31, 33, 127, 128, 129, 257, 1023, 1024, 1025, 1281, 2049, 5000]


def shapes(n, seed):
    from sequoia_gb300 import scenes
    soup = scenes.gaussian_soup(n, 3, seed=seed)
    line = soup.copy()
    line[:, 0::3] += np.repeat(np.exp2(np.linspace(0, 20, n)).astype(np.float32)[:, None], 3, 1)  # one split peels few
    same = soup.copy()
    same[n // 3:] = soup[0]  # most centroids coincide
    return {"soup": soup, "line": line, "same": same}


@pytest.mark.parametrize("bins,leaf", [(8, 8), (5, 1), (16, 4), (12, 2), (32, 1)])
@pytest.mark.parametrize("n", SIZES)
def test_sah_phase_edges(ctx, oracle, n, bins, leaf):
    for name, tris in shapes(n, 900 + n).items():
        bvh = ctx.build(tris, "sah", bins=bins, leaf=leaf)
        nodes, root = bvh.export_node1()
        onodes, oroot, _ = oracle.build_sah(tris, bins, leaf)
        assert_same_tree(oracle, nodes, root, onodes, oroot)
        assert (oracle.leaf_reach(nodes, root, n) == 1).all(), name
    assert ctx.sync() == 0
