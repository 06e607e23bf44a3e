"""The refit by blocks of sorted slots at the edges of its blocks, and on trees
cut at the stack's depth, whose leaves hold many boxes and cross blocks,
against the oracle bit for bit."""

import numpy as np
import pytest

import phiray_b200 as px
from tests import gen
from tests.test_gpu_bvh import same_tree

pytestmark = pytest.mark.gpu


def deep_prims(n: int, seed: int) -> np.ndarray:
    """Boxes at halving distances from the origin and many within the last
    cell: equal codes under a chain of some thirty inner nodes."""
    rng = np.random.default_rng(seed)
    c = np.full((n, 3), 2.0 ** -14)
    c[: n // 8] = 2.0 ** -rng.integers(0, 12, size=(n // 8, 3))
    h = rng.uniform(0.0, 2.0 ** -15, size=(n, 3))
    p = np.zeros((n, 8), np.float32)
    p[:, 0:3], p[:, 4:7] = c - h, c + h
    return p[rng.permutation(n)]


@pytest.mark.parametrize("n,leaf,deep", [(511, 1, False), (512, 4, False), (513, 1, False), (1025, 2, False),
                                         (1537, 3, False), (700, 1, True), (20_000, 4, True), (5_000, 8, True)])
def test_refit_at_block_edges(gpu, orc, n, leaf, deep):
    p = deep_prims(n, n) if deep else gen.bvh_prims(n, 0.0)
    nodes, order, depth = orc.build(p, leaf)
    if deep:
        cut = nodes.view(np.uint32)[orc.reachable(nodes)]
        cut = cut[cut[:, 3] >> 31 == 1]
        assert np.max(cut[:, 7] - (cut[:, 3] & 0x7FFFFFFF)) > leaf  # a leaf the depth cut short
    g = px.GpuBvh.build(gpu, p, leaf)
    same_tree(g.download(), nodes, order, depth, orc)
    moved = p.copy()
    moved[:, [0, 1, 2, 4, 5, 6]] += np.random.default_rng(1).normal(size=(n, 1)).astype(np.float32)
    assert g.update(moved)
    want = orc.refit(nodes, order, moved)
    same_tree(g.download(), want, order, depth, orc)
    g.refit()
    same_tree(g.download(), want, order, depth, orc)
