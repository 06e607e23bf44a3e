"""The one-block build of small trees at the edges of its warps' runs, its
rounds of threads and its range, with deep trees and equal codes, against the
oracle bit for bit; and a refit of what it built."""

import numpy as np
import pytest

import phiray_b200 as px
from tests import gen
from tests.test_gpu_bvh import same_tree
from tests.test_gpu_refit_blocks import deep_prims

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,leaf,kind", [(1, 1, "grid"), (31, 1, "grid"), (33, 4, "grid"), (256, 1, "same"),
                                         (1024, 2, "grid"), (1025, 1, "deep"), (2049, 8, "grid"), (3001, 3, "deep"),
                                         (4095, 1, "same"), (4096, 4, "grid"), (4097, 4, "grid")])
def test_small_build_and_refit(gpu, orc, n, leaf, kind):
    p = deep_prims(n, n) if kind == "deep" else gen.bvh_prims(n, 0.0)
    if kind == "same":
        p[:] = p[0]  # equal codes: the links follow the indices
    nodes, order, depth = orc.build(p, leaf)
    g = px.GpuBvh.build(gpu, p, leaf)
    same_tree(g.download(), nodes, order, depth, orc)
    moved = p.copy()
    moved[:, [0, 1, 2, 4, 5, 6]] += np.random.default_rng(n).normal(size=(n, 1)).astype(np.float32)
    for _ in range(2):
        assert g.update(moved)
        same_tree(g.download(), orc.refit(nodes, order, moved), order, depth, orc)
