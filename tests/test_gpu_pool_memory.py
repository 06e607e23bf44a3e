"""The pooled render's memory follows the frame."""

import pytest

import phiray_b200 as px
from phiray_b200 import scenes
from tests.test_gpu_trace import cam_of

pytestmark = pytest.mark.gpu


def test_a_small_frame_reserves_little():
    import torch

    torch.zeros(1, device="cuda")
    gpu = px.Gpu(0)  # a context of its own: its pool keeps what it ever held
    s = scenes.c2_mesh(levels=4, width=64, height=48)
    tr = px.Tracer.of(gpu, s)
    cam = cam_of(s, 64, 48)
    tr.set_kernel(px.Tracer.MEGAKERNEL)
    tr.trace(cam, 64, 48, 0, 1)
    gpu.wait()
    before = torch.cuda.mem_get_info()[0]
    tr.set_kernel(px.Tracer.STATE_MACHINE)
    tr.trace(cam, 64, 48, 0, 1)
    gpu.wait()
    # 32 slots of 244 bytes for each block, 40 bytes a sample, and the pool's steps of 32 MB
    assert before - torch.cuda.mem_get_info()[0] <= 72 << 20
    tr.close()
    gpu.close()
