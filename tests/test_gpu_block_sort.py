"""One-block radix sort: every pass of a small sort runs in one block's shared
memory (8 keys per thread, at least eight warps), against a stable argsort."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# warp runs of 256 keys, the smallest block (2,048 keys), the largest sort of
# one block (8,192) and the first of the tile kernels
@pytest.mark.parametrize("n", [1, 31, 33, 256, 257, 2047, 2049, 8191, 8192, 8193])
@pytest.mark.parametrize("key_bits,digit_bits", [(32, 6), (32, 8), (32, 10), (9, 8), (3, 6)])
def test_small_sorts_are_stable(ctx, n, key_bits, digit_bits):
    rng = np.random.default_rng(n * 100 + key_bits + digit_bits)
    keys = rng.integers(0, 1 << key_bits, n, dtype=np.uint64).astype(np.uint32)
    keys[n // 2:] = keys[n // 2]  # long runs of one digit
    keys[-1] = (1 << key_bits) - 1
    vals = rng.permutation(n).astype(np.uint32)
    k, v = ctx.radix_sort_pairs(keys, vals, key_bits, digit_bits)
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(k, keys[order])
    assert np.array_equal(v, vals[order])
    assert ctx.sync() == 0


def test_one_block_sort_builds_the_oracles_trees(ctx, oracle):
    """Builds at the limit: 30-bit codes, and 60-bit codes (two sorts in turn)."""
    from sequoia_gb300 import scenes
    for n in (2, 8192, 8193):
        tris = scenes.gaussian_soup(n, 8, seed=n)
        onodes, oroot, _, _ = oracle.build_morton(tris)
        want = oracle.canonical_bfs(onodes, oroot)
        bvh = ctx.build(tris, "morton")
        nodes, root = bvh.export_node1()
        assert np.array_equal(oracle.canonical_bfs(nodes, root)["child"], want["child"])
        bvh.free()
        bvh = ctx.build(tris, "morton", morton64=True)
        codes, perm = bvh.export_sorted64()
        assert np.all(codes[:-1] <= codes[1:]) and np.array_equal(np.sort(perm), np.arange(n))
        same = codes[:-1] == codes[1:]
        assert np.all(perm[:-1][same] < perm[1:][same])
        bvh.free()
