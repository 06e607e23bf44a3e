"""Pooled frames of several launches (more samples than the buffer of terms
holds) are the megakernel's, word for word."""

import numpy as np
import pytest

import phiray_b200 as px
from phiray_b200 import scenes
from tests.test_gpu_trace import cam_of

pytestmark = pytest.mark.gpu


# 1080p holds 12 samples' terms in a launch: 13 run as 7 + 6, 25 as 9 + 9 + 7
@pytest.mark.parametrize("spp,kernel", [(13, px.Tracer.STATE_MACHINE), (25, px.Tracer.STATE_MACHINE_6)])
def test_frames_of_several_launches_equal_the_megakernel(gpu, spp, kernel):
    s = scenes.c2_mesh(levels=5, width=1920, height=1080, bounces=2)
    cam = cam_of(s, 1920, 1080)
    images, rays = [], []
    for k in (px.Tracer.MEGAKERNEL_16_SYNC, kernel):
        tr = px.Tracer.of(gpu, s)
        tr.set_kernel(k)
        tr.trace(cam, 1920, 1080, 0, spp)
        images.append(tr.image())
        rays.append(tr.time()[1])
        tr.close()
    assert np.array_equal(images[0], images[1]) and rays[0] == rays[1]
