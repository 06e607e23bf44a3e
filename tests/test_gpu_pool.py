"""The pooled render == the megakernel, word for word, at the frame sizes and
sample counts where its units, pools and launches have edges (the megakernel
itself is held to the oracle in test_gpu_trace.py)."""

import numpy as np
import pytest

import phiray_b200 as px
from phiray_b200 import scenes
from tests import oracle_lib
from tests.test_gpu_trace import cam_of, check_image

pytestmark = pytest.mark.gpu

POOLED = [px.Tracer.STATE_MACHINE, px.Tracer.STATE_MACHINE_6, px.Tracer.STATE_MACHINE_8, None]


# one pixel; part of a tile; tiles and a rest; warp tiles (sides multiples of
# 16 and 8); more units than the pools' slots
@pytest.mark.parametrize("w,h,spp", [(1, 1, 1), (33, 1, 3), (37, 23, 5), (64, 48, 17), (640, 360, 8)])
def test_pooled_render_equals_megakernel(gpu, w, h, spp):
    s = scenes.c2_mesh(levels=5, width=w, height=h)
    cam = cam_of(s, w, h)
    tr = px.Tracer.of(gpu, s)
    tr.set_kernel(px.Tracer.MEGAKERNEL)
    tr.trace(cam, w, h, 0, spp)
    want, rays = tr.image(), tr.time()[1]
    tr.close()
    for kernel in POOLED:
        tr = px.Tracer.of(gpu, s)
        if kernel is not None:
            tr.set_kernel(kernel)
        # in two calls: the second adds to the first's sums
        tr.trace(cam, w, h, 0, max(spp // 2, 1))
        n = tr.time()[1]
        if spp > 1:
            tr.trace(cam, w, h, spp // 2, spp - spp // 2)
            n += tr.time()[1]
        assert np.array_equal(tr.image(), want), kernel
        assert n == rays
        tr.close()


@pytest.mark.parametrize("kind", ["glass", "cutout", "layers", "lamps", "rig"])
def test_pooled_render_of_every_material(gpu, kind):
    # glass transmits: the pooled ids fall back to the megakernel there
    s = scenes.features(kind) if kind != "cutout" else scenes.c1_plain(ntris=500, width=48, height=40, spp=6)
    if kind == "cutout":
        s.mats[::3, 3] = 0.4  # every third face lets most camera rays pass
    cam = cam_of(s, s.width, s.height)
    images = []
    for kernel in [px.Tracer.MEGAKERNEL, *POOLED]:
        tr = px.Tracer.of(gpu, s)
        if kernel is not None:
            tr.set_kernel(kernel)
        tr.trace(cam, s.width, s.height, 0, 6)
        images.append(tr.image())
        tr.close()
    assert all(np.array_equal(images[0], i) for i in images[1:])


def test_pooled_render_of_rows_and_a_tree_that_is_one_leaf(gpu):
    s = scenes.c1_plain(ntris=2, width=50, height=30, spp=4)
    cam = cam_of(s, 50, 30)
    images = []
    for kernel in (px.Tracer.MEGAKERNEL, px.Tracer.STATE_MACHINE):
        tr = px.Tracer.of(gpu, s, leaf=16)
        tr.set_kernel(kernel)
        lib = px.lib()
        for row, rows in ((0, 7), (7, 23)):
            assert lib.phx_tracer_trace_rows(tr.handle, cam.ctypes.data, 50, 30, 0, 4, row, rows) == 0
        images.append(tr.image())
        tr.close()
    assert np.array_equal(images[0], images[1])


# no emitter in a run of slots, one, runs full of them; a rest of a run
@pytest.mark.parametrize("ntris,every", [(1500, 1), (3000, 700), (2047, 2047)])
def test_emitter_table(gpu, orc, ntris, every):
    s = scenes.c1_plain(ntris=ntris, width=32, height=24, spp=2)
    s.mats[:ntris:every, 8:11] = 0.5
    cam = cam_of(s, 32, 24)
    want, rays = oracle_lib.TraceOracle(orc, s).trace(cam, 0, 2)
    tr = px.Tracer.of(gpu, s)
    tr.trace(cam, 32, 24, 0, 2)
    check_image(tr.image(), want, 32 * 24)
    assert tr.time()[1] == rays
    tr.close()
