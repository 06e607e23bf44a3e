"""The pooled render near the device's memory: its buffers go to an allocation
that finds none, and frames without them are the megakernel's."""

import numpy as np
import pytest

import phiray_b200 as px
from phiray_b200 import scenes
from tests.test_gpu_trace import cam_of

pytestmark = pytest.mark.gpu


def test_pooled_buffers_give_way_to_other_allocations():
    import torch

    torch.zeros(1, device="cuda")
    torch.cuda.empty_cache()
    s = scenes.c2_mesh(levels=4, width=1280, height=720)
    cam = cam_of(s, 1280, 720)
    gpu = px.Gpu(0)
    tr = px.Tracer.of(gpu, s)
    tr.set_kernel(px.Tracer.MEGAKERNEL_16_SYNC)
    tr.trace(cam, 1280, 720, 0, 12)
    want = tr.image()
    # all but 3 GB of the device taken (not written)
    hog = torch.empty(torch.cuda.mem_get_info()[0] - (3 << 30), dtype=torch.uint8, device="cuda")
    tr.set_kernel(px.Tracer.STATE_MACHINE)
    tr.trace(cam, 1280, 720, 0, 12)  # 0.44 GB of terms and 0.3 of paths
    assert np.array_equal(tr.image(), want)
    gpu.wait()
    room = torch.cuda.mem_get_info()[0]
    big = px.GpuArray(gpu, room + (256 << 20))  # fits once they are given back
    tr.trace(cam, 1280, 720, 0, 12)
    assert np.array_equal(tr.image(), want)
    # the same frame where there is no room for the buffers at all
    rest = torch.empty(max(torch.cuda.mem_get_info()[0] - (160 << 20), 1 << 20), dtype=torch.uint8, device="cuda")
    tr.trace(cam, 1280, 720, 0, 12)
    assert np.array_equal(tr.image(), want)
    with pytest.raises(px.PhxError):
        px.GpuArray(gpu, 8 << 30)
    tr.trace(cam, 1280, 720, 0, 12)  # and the context goes on
    assert np.array_equal(tr.image(), want)
    del hog, rest
    big.free()
    tr.close()
    gpu.close()
    torch.cuda.empty_cache()
