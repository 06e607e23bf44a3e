"""The pooled render == the megakernel over the forms of frames that it takes:
materials, world, lights, camera and limits drawn at random, their extremes
among them (black and lit worlds, the studio rig, no and every light, cut-outs,
metals that would transmit, indices of refraction at and below one)."""

import numpy as np
import pytest

import phiray_b200 as px
from phiray_b200 import scenes
from tests.test_gpu_trace import cam_of

pytestmark = pytest.mark.gpu


def _scene(rng):
    kind = rng.choice(["lamps", "rig", "layers", "cloud", "mesh"])
    if kind in ("lamps", "rig", "layers"):
        s = scenes.features(str(kind))
    elif kind == "cloud":
        s = scenes.c1_plain(ntris=int(rng.integers(3, 900)), width=48, height=40, spp=1)
    else:
        s = scenes.c2_mesh(levels=3, width=48, height=40)
    m = s.mats  # (words as scenes.mat lays them out)
    n = len(m)

    def some(values, at, share=0.5):
        hit = rng.random(n) < share
        m[hit, at] = rng.choice(values, int(hit.sum()))

    some([0.0, 0.4, 0.9], 3, 0.3)              # opacity
    some([0.0, 0.02, 0.3, 1.0, 2.0], 4)        # roughness
    some([0.0, 0.5, 1.0], 5)                   # metal
    m[:, 6] = np.where(m[:, 5] == 1.0, rng.choice([0.0, 1.0], n), 0.0)  # a whole metal transmits nothing
    some([0.7, 1.0, 1.0001, 1.5, 2.4], 7)      # index of refraction
    some([0.0, 0.6, 1.0], 17, 0.3)             # subsurface
    some([0.0, 1.0], 21, 0.3)                  # sheen
    some([0.0, 0.5, 1.0], 26, 0.3)             # coat
    if rng.random() < 0.4:
        lit = rng.random(n) < 0.1
        m[lit, 8:11] = rng.choice([0.5, 5.0, 1e4], (int(lit.sum()), 3))
    return s


def _camera(rng, s, w, h):
    c = cam_of(s, w, h)
    c["env"][0, :3] = rng.choice([0.0, 0.05, 1.0, -0.1]) * rng.random(3)
    if rng.random() < 0.4:
        c["count"] = rng.integers(0, int(c["count"][0]) + 1)
    c["bounces"] = rng.choice([0, 1, 2, 8, 40])
    c["ao"] = rng.choice([0.0, 0.05, 10.0])
    c["limit"][0, :2] = rng.choice([0.0, 0.5, 10.0], 2)
    c["sky"] = rng.random(4).astype(np.float32)
    c["pan"] = rng.uniform(-0.2, 0.2, 2).astype(np.float32)
    c["persp"] = int(rng.random() < 0.8)
    c["view"][0, 1:3] = (rng.choice([0.0, 1.0]), rng.choice([1.0, 2.2]))
    return c


@pytest.mark.parametrize("seed", range(24))
def test_pooled_render_equals_megakernel_over_its_forms(gpu, seed):
    rng = np.random.default_rng(seed)
    s = _scene(rng)
    w, h, spp = int(rng.integers(1, 70)), int(rng.integers(1, 60)), int(rng.integers(1, 9))
    cam = _camera(rng, s, w, h)
    first = int(rng.choice([0, 0, 7]))
    images, rays = [], []
    for kernel in (px.Tracer.MEGAKERNEL, px.Tracer.STATE_MACHINE, px.Tracer.STATE_MACHINE_8):
        tr = px.Tracer.of(gpu, s, leaf=int(1 + seed % 5))
        if seed % 3 == 0:
            tr.set_tree(px.Tracer.TREE_SAH)
        tr.set_kernel(kernel)
        tr.trace(cam, w, h, first, spp)
        images.append(tr.image())
        rays.append(tr.time()[1])
        tr.close()
    assert all(np.array_equal(images[0], i) for i in images[1:])
    assert rays[0] == rays[1] == rays[2]
