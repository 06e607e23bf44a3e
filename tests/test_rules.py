"""The host's decisions between paths (phiray_b200/csrc/rules.cuh), built for
the host: which calls take which path, over the forms that they accept. And the
index arithmetic of the convolutions' copies (conv_index.cuh)."""

import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

from phiray_b200.tracer import Tracer

HERE = Path(__file__).resolve().parent


@pytest.fixture(scope="module")
def rules(tmp_path_factory):
    out = tmp_path_factory.mktemp("rules") / "librules.so"
    subprocess.run(["g++", "-O1", "-std=c++17", "-shared", "-fPIC", "-Wall", "-Werror", "-o", str(out),
                    str(HERE / "rules_probe.cpp")], check=True)
    return C.CDLL(str(out))


def test_wide_accesses_only_at_their_alignment(rules):
    rules.probe_aligned16.argtypes = [C.c_void_p]
    for p in range(0x7F0000000000, 0x7F0000000000 + 64):
        assert rules.probe_aligned16(p) == (p % 16 == 0)


FULL, ADAPTIVE, TRANSMITS, CAPTURING = 1, 2, 4, 8
POOLED = (Tracer.STATE_MACHINE, Tracer.STATE_MACHINE_6, Tracer.STATE_MACHINE_8)
UNSET = 0xFFFFFFFF


# one sample and many, around the sizes where the default changes
FRAMES = [(64, 1, 12), (99_999, 1, 9_999), (100_000, 1, 9_999), (99_999, 1, 10_000), (64, 2, 12), (299_999, 1, 50_000),
          (300_000, 1, 50_000), (2_073_600, 1, 12), (65_536, 16, 65_540), (2_073_600, 64, 1_310_722)]


@pytest.mark.parametrize("mega", [Tracer.MEGAKERNEL, Tracer.MEGAKERNEL_16_SYNC])
@pytest.mark.parametrize("flags", range(16))
def test_every_frame_has_a_kernel_that_can_trace_it(rules, flags, mega):
    rules.probe_frame_kernel.restype = C.c_uint32
    for kernel in [*range(Tracer.KERNELS), UNSET]:
        for pixels, spp, faces in FRAMES:
            r = rules.probe_frame_kernel(C.c_uint32(kernel), mega, flags, pixels, spp, faces)
            got, buffers = r & 0x7FFFFFFF, bool(r >> 31)
            wavefront_can = not flags & (ADAPTIVE | CAPTURING)
            pooled_can = not flags & ADAPTIVE and (flags & FULL or not flags & TRANSMITS)
            if kernel == UNSET:
                brief = spp == 1 and pixels < 100_000 and faces < 10_000
                form = Tracer.STATE_MACHINE_6 if pixels * spp < 300_000 else Tracer.STATE_MACHINE
                want = form if pooled_can and not flags & FULL and not brief else mega
            elif kernel == Tracer.WAVEFRONT and not wavefront_can or kernel in POOLED and not pooled_can:
                want = mega
            else:
                want = kernel
            assert got == want
            assert buffers == (got in POOLED and not flags & FULL)


def test_autotuning_keeps_the_fastest_megakernel_beside_its_pick(rules):
    """A tracer whose fastest kernel is the pooled render traces its adaptive
    frames with the fastest megakernel form, not with the 4-block one."""
    rng = np.random.default_rng(5)
    others = {*POOLED, Tracer.WAVEFRONT}
    for _ in range(50):
        ms = rng.uniform(1.0, 9.0, Tracer.KERNELS).astype(np.float32)
        ms[list(others)] -= 5.0
        got = rules.probe_fastest_megakernel(ms.ctypes.data_as(C.c_void_p))
        assert got not in others and ms[got] == min(ms[k] for k in range(Tracer.KERNELS) if k not in others)


def test_of_pooled_forms_close_together_the_largest_blocks(rules):
    def pick(*pooled, mega=9.0):
        ms = np.full(Tracer.KERNELS, 9.0, np.float32)
        ms[list(POOLED)], ms[15] = pooled, mega
        return rules.probe_autotuned(ms.ctypes.data_as(C.c_void_p), int(np.argmin(ms)))

    assert pick(2.71, 2.67, 2.83) == 1
    assert pick(2.84, 2.67, 2.83) == 2  # 512 threads 6.4 % behind
    assert pick(1.87, 2.12, 1.50) == 3
    assert pick(2.5, 2.6, 2.7) == 1
    assert pick(2.71, 2.67, 2.83, mega=2.0) == 15


@pytest.mark.parametrize("fails", [0, 1, 2, 99])
@pytest.mark.parametrize("seed", range(6))
def test_lanes_reserve_once_for_their_pooled_jobs(rules, seed, fails):
    """A lane's buffers are asked for once, before its first launch, for the
    largest need of its pooled jobs; where that fails none of its jobs has any."""
    rng = np.random.default_rng(seed)
    n, lanes = int(rng.integers(1, 12)), 3
    jobs = np.zeros((n, 4), np.uint64)
    jobs[:, 0] = rng.integers(1, 1000, n)
    jobs[:, 1] = rng.integers(0, 2, n) if seed else 0  # (seed 0: none runs pooled)
    # the larger job need not be the one with the larger buffers
    jobs[:, 2:] = rng.integers(1, 1000, (n, 2))
    calls, order, lane = np.zeros((8, 3), np.uint64), np.zeros(n, np.uint32), np.zeros(n, np.uint32)
    buffers = np.zeros(n, np.uint8)
    made = rules.probe_lanes(*(a.ctypes.data_as(C.c_void_p) if isinstance(a, np.ndarray) else a
                               for a in (jobs, n, lanes, fails, calls, order, lane, buffers)))
    assert sorted(order) == list(range(n)) and (np.diff(jobs[order, 0].astype(int)) <= 0).all()
    assert (lane < lanes).all()
    calls = calls[:made]
    assert len(set(calls[:, 0])) == made  # once a lane
    for k in range(lanes):
        mine = (lane == k) & (jobs[:, 1] != 0)
        at = np.flatnonzero(calls[:, 0] == k)
        assert len(at) == int(mine.any())
        if mine.any():
            assert (calls[at[0], 1:] == jobs[mine, 2:].max(0)).all()
            assert (buffers[mine] == (at[0] != fails)).all()
    assert not buffers[jobs[:, 1] == 0].any()


@pytest.mark.parametrize("count", [1, 33, 64 * 48, 256 * 256, 1920 * 1080, 2400 * 1800, 120_000_000])
@pytest.mark.parametrize("spp", [1, 3, 7, 13, 16, 64, 4000])
@pytest.mark.parametrize("blocks,most", [(296, 4096), (592, 2048), (1184, 1024), (2, 4096)])
def test_pooled_render_memory_follows_the_frame(rules, count, spp, blocks, most):
    plan = (C.c_uint64 * 5)()
    first = rules.probe_pool_plan(count, spp, blocks, most, 1, plan)
    got_blocks, slots, per, state, out = plan
    assert got_blocks == blocks and 32 <= slots <= most and slots % 32 == 0
    assert 1 <= per <= spp and out == count * per * 40
    assert out <= max(1 << 30, count * 40)
    # all blocks' slots, no more than the frame has paths (or a group of 32 each)
    assert state == blocks * slots * 244
    assert blocks * slots <= max(count * per, 32 * blocks)
    left = spp
    while left:  # no launch takes more slots than the plan holds
        now = min(left, per)
        assert 32 <= rules.probe_pool_plan(count, spp, blocks, most, now, plan) <= slots
        left -= now
    assert 32 <= first <= slots
    assert -(-spp // per) == -(-spp // min(max((1 << 30) // (count * 40), 1), spp))  # as many launches as it takes


# 15.8 M pixels wide is where (row W + column) 8 passes 2^31, 126 M where row W does
@pytest.mark.parametrize("width", [1, 8, 1920, 15_790_320, 15_800_000, 67_108_864, 126_000_000])
@pytest.mark.parametrize("groups", [2, 4, 6, 8])
def test_patch_vectors_of_wide_images(rules, width, groups):
    PX, PY = 10, 18
    lbo, seen = PX * PY * 16, set()
    out = (C.c_int64 * 5)()
    for v in range(PX * PY * groups):
        rules.probe_patch_vec(v, groups, PX, lbo, width, out)
        q, g = divmod(v, groups)
        row, col = divmod(q, PX)
        assert list(out) == [row * width + col, g * lbo + q * 16, 8 * g, row, col]
        seen.add(out[1])
    assert len(seen) == PX * PY * groups
