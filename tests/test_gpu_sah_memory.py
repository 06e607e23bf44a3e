"""The SAH build's scratch: no more a box than the level-by-level build took
(160 bytes), so that what fitted the device then fits now."""

import ctypes as C

import pytest

import phiray_b200 as px
from phiray_b200 import _native as N

pytestmark = pytest.mark.gpu


def test_sah_build_scratch_a_box():
    import torch

    n = 4_000_000
    g = torch.Generator(device="cuda").manual_seed(1)
    prims = torch.zeros(n, 8, device="cuda")
    prims[:, 0:3] = torch.rand(n, 3, generator=g, device="cuda")
    prims[:, 4:7] = prims[:, 0:3] + 0.01
    nodes, order = torch.zeros(2 * n, 8, device="cuda"), torch.zeros(n, dtype=torch.int32, device="cuda")
    gpu = px.Gpu(0)  # a context of its own: its pool keeps what it ever held
    count, depth = C.c_uint32(), C.c_uint32()

    def build(m):
        N.check(px.lib().phx_bvh_build_sah(gpu.handle, prims.data_ptr(), m, 4, nodes.data_ptr(), order.data_ptr(),
                                           C.byref(count), C.byref(depth)))

    build(5000)  # the kernels' code is loaded
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    build(n)
    # (the pool grows in steps of 32 MB)
    assert before - torch.cuda.mem_get_info()[0] <= 160 * n + (64 << 20)
    gpu.close()
