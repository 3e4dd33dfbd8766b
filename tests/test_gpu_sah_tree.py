"""The one-CTA tree builder at the sizes where its parts meet, bit for bit
(0 ulp) against the oracle's builder: trees of one and two prims, around a
warp, around the size above which the whole CTA splits a node, several rounds
of the CTA, and past the largest tree of one CTA (built level by level)."""
import numpy as np
import pytest

import vrg
from helpers import first_node_diff, gpu_build_bl, gpu_build_tl, nodes_equal, random_aabbs, random_tris

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 3, 4, 9, 10, 11, 12, 31, 32, 33, 65, 255, 256, 257, 258, 511, 513, 1023, 1300, 4099]


def _check(got, ref, n):
    nodes, order = got
    rn, ro = ref[0], ref[1]
    assert np.array_equal(order, np.asarray(ro, np.uint32)), n
    assert nodes_equal(nodes, rn.view(vrg.NODE_DTYPE).reshape(nodes.shape)), (n, first_node_diff(nodes, rn))


@pytest.mark.parametrize("kind", ["grid", "random", "same", "line"])
def test_tree_sizes(gpu_ctx, orc, kind):
    rng = np.random.default_rng(5)
    sets = []
    for n in SIZES:
        if kind == "same":    # no plane separates: halves in the current order
            a = np.tile(np.array([[1, 2, 3, 2, 3, 4]], np.float32), (n, 1))
        elif kind == "line":  # one axis, many equal centroids
            x = rng.integers(0, 7, n).astype(np.float32)
            a = np.stack([x, 0 * x, 0 * x, x + 1, 0 * x + 1, 0 * x + 1], 1).astype(np.float32)
        else:
            a = random_aabbs(rng, n, grid=kind == "grid")
        sets.append((a, (rng.random(n) * 10).astype(np.float32), rng.permutation(n).astype(np.uint32), None))
    for s, got in zip(sets, gpu_build_tl(gpu_ctx, sets)):
        _check(got, orc.build_tl_bvh(s[0], s[1], s[2]), len(s[0]))


def test_triangle_trees(gpu_ctx, orc):
    rng = np.random.default_rng(6)
    sets = [(random_tris(rng, n), (rng.random(n) * 5).astype(np.float32), np.arange(n, dtype=np.uint32))
            for n in (1, 2, 3, 70, 300, 2000)]
    for s, got in zip(sets, gpu_build_bl(gpu_ctx, sets)):
        _check(got, orc.build_bl_bvh(*s), len(s[0]))


def test_largest_tree_of_a_cta_beside_larger_ones(gpu_ctx, orc):
    rng = np.random.default_rng(7)
    sets = []
    for n in (2560, 2561, 300, 9000):
        a = random_aabbs(rng, n, scale=900.0)
        sets.append((a, (rng.random(n) * 3).astype(np.float32), np.arange(n, dtype=np.uint32), None))
    for s, got in zip(sets, gpu_build_tl(gpu_ctx, sets)):
        _check(got, orc.build_tl_bvh(s[0], s[1], s[2]), len(s[0]))
