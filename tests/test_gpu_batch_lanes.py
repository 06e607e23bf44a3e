"""The batch launched scene by scene: tracers of every kernel beside one
another give their own images, and the side streams hold memory only for
launches that use it."""

import numpy as np
import pytest

import phiray_b200 as px
from phiray_b200 import scenes
from phiray_b200.batch import PER_SCENE, PERSISTENT, Batch
from tests.test_gpu_batch import _jobs, _single

pytestmark = pytest.mark.gpu


def _batch(gpu, jobs, kernels):
    tracers, b = [], Batch(gpu)
    for (s, cam, first), kernel in zip(jobs, kernels):
        t = px.Tracer.of(gpu, s)
        if kernel is not None:
            t.set_kernel(kernel)
        tracers.append(t)
        b.add(t, cam, s.width, s.height, first, s.spp)
    b.set_config(PER_SCENE)
    return b, tracers


def _close(b, tracers):
    b.close()
    for t in tracers:
        t.close()


def test_tracers_of_different_kernels_in_one_batch(gpu):
    jobs = [*_jobs(), *((s, cam, 0) for s, cam, _ in _jobs())]
    want = _single(gpu, jobs)
    kernels = [None, px.Tracer.WAVEFRONT, px.Tracer.STATE_MACHINE_8, px.Tracer.MEGAKERNEL_16_SYNC,
               px.Tracer.WAVEFRONT, None, px.Tracer.MEGAKERNEL, px.Tracer.STATE_MACHINE_6]
    b, tracers = _batch(gpu, jobs, kernels)
    for again in range(2):
        b.trace()
        for k, (t, w) in enumerate(zip(tracers, want)):
            if not again or jobs[k][2] == 0:  # (a frame from a later sample on adds to what is there)
                assert np.array_equal(t.image(), w), (again, k)
    _close(b, tracers)


def _free():
    import torch

    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def test_lanes_hold_memory_only_for_pooled_launches():
    import torch

    torch.zeros(1, device="cuda")
    gpu = px.Gpu(0)  # a context of its own: its pool keeps what it ever held
    b, tracers = _batch(gpu, _jobs(), [px.Tracer.MEGAKERNEL, px.Tracer.MEGAKERNEL_16_SYNC, px.Tracer.MEGAKERNEL_8,
                                       px.Tracer.WAVEFRONT])
    gpu.wait()
    before = _free()
    b.trace()
    gpu.wait()
    # the wavefront's slots for 1,280 pixels and its queues
    assert before - _free() <= 64 << 20
    b.set_config(PERSISTENT)
    b.trace()
    gpu.wait()
    assert before - _free() <= 64 << 20
    _close(b, tracers)
    gpu.close()
