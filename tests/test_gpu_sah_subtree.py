"""The SAH build's subtree and partition paths at their edges == the
restatement of Bvh::build_sah, word for word."""

import numpy as np
import pytest

from phiray_b200.bvh import build_sah

pytestmark = pytest.mark.gpu


def _boxes(n, kind):
    rng = np.random.default_rng(n)
    p = np.zeros((n, 8), np.float32)
    lo = rng.uniform(-1.0, 1.0, (n, 3)).astype(np.float32)
    if kind == "line":  # one axis with planes
        lo[:, 1:] = 0.25
    elif kind == "grid":  # many equal costs and shared bins
        lo = np.round(lo * 2.0) / 2.0
    elif kind == "outliers":  # splits of a few slots against the rest, at many scales
        lo *= np.exp(-rng.uniform(0.0, 12.0, (n, 1))).astype(np.float32)
        lo[::n // 3 + 1] += 1e6
    elif kind == "nan":  # bounds that are not numbers lose
        lo[::5, 1] = np.nan
    p[:, 0:3], p[:, 4:7] = lo, lo + rng.uniform(0.0, 0.1, (n, 3)).astype(np.float32)
    return p


# a word of a subtree's mask and its ends (32), a whole subtree (127), the
# first sizes that are a block's (128), two chunks of the partition
@pytest.mark.parametrize("n", [31, 32, 33, 64, 65, 127, 128, 129, 511, 4097])
@pytest.mark.parametrize("kind", ["line", "grid", "outliers", "nan"])
@pytest.mark.parametrize("leaf", [1, 4, 200])
def test_sah_build_equals_the_reference_tree(gpu, orc, n, kind, leaf):
    p = _boxes(n, kind)
    want_nodes, want_order, want_depth = orc.build_sah(p, leaf)
    got = build_sah(gpu, p, leaf)
    assert got.depth == want_depth
    assert np.array_equal(got.order, want_order)
    assert np.array_equal(got.nodes.view(np.uint32), want_nodes.view(np.uint32))


def test_partition_chains_longer_than_a_round(gpu, orc):
    """A node whose right slots come first: every left slot rotates the
    queue, so a log entry's chain runs through thousands of links."""
    n = 20000
    rng = np.random.default_rng(3)
    p = np.zeros((n, 8), np.float32)
    lo = rng.uniform(0.0, 0.01, (n, 3)).astype(np.float32)
    lo[:3, 0] += 50.0  # three right slots, then lefts
    p[:, 0:3], p[:, 4:7] = lo, lo + np.float32(0.001)
    want_nodes, want_order, want_depth = orc.build_sah(p, 4)
    got = build_sah(gpu, p, 4)
    assert got.depth == want_depth and np.array_equal(got.order, want_order)
    assert np.array_equal(got.nodes.view(np.uint32), want_nodes.view(np.uint32))
