"""The SAH build over arrays that start inside a packed buffer, at addresses
that are multiples of 4 bytes only == the same build over whole buffers."""

import ctypes as C

import numpy as np
import pytest

import phiray_b200 as px
from phiray_b200 import _native as N

pytestmark = pytest.mark.gpu


# a subtree alone, one of a block's nodes above it, the chunked levels
@pytest.mark.parametrize("n", [1, 100, 700, 5000])
@pytest.mark.parametrize("prims_at,nodes_at", [(1, 0), (0, 3), (2, 1)])
def test_sah_build_in_a_packed_buffer(gpu, orc, n, prims_at, nodes_at):
    import torch

    rng = np.random.default_rng(n)
    p = np.zeros((n, 8), np.float32)
    lo = rng.uniform(-1.0, 1.0, (n, 3)).astype(np.float32)
    p[:, 0:3], p[:, 4:7] = lo, lo + rng.uniform(0.0, 0.1, (n, 3)).astype(np.float32)
    want_nodes, want_order, want_depth = orc.build_sah(p, 4)
    prims = torch.zeros(prims_at + 8 * n, device="cuda")
    prims[prims_at:] = torch.from_numpy(p.reshape(-1))
    nodes = torch.zeros(nodes_at + 8 * (2 * n - 1), device="cuda")
    order = torch.zeros(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    count, depth = C.c_uint32(), C.c_uint32()
    N.check(px.lib().phx_bvh_build_sah(gpu.handle, prims[prims_at:].data_ptr(), n, 4,
                                       nodes[nodes_at:].data_ptr(), order.data_ptr(), C.byref(count),
                                       C.byref(depth)))
    got = nodes[nodes_at:].cpu().numpy().reshape(-1, 8)[: count.value]
    assert depth.value == want_depth
    assert np.array_equal(order.cpu().numpy().view(np.uint32), want_order)
    assert np.array_equal(got.view(np.uint32), want_nodes.view(np.uint32))
    assert not nodes[:nodes_at].any() and np.array_equal(prims[prims_at:].cpu().numpy(), p.reshape(-1))
