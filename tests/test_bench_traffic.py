"""The DRAM traffic that the benchmark reports beside a frame: only that of the
kernel, size and sample count it was captured with."""

import bench


def test_traffic_is_reported_for_what_was_captured_only():
    pooled = [k for k, n in enumerate(bench.KERNEL_NAMES) if n.startswith("pooled")]
    bytes_of = {k: bench.frame_traffic(k, 1920, 1080, 64) for k in range(len(bench.KERNEL_NAMES))}
    assert [k for k, b in bytes_of.items() if b is not None] == pooled
    for k in pooled:
        # the terms of every sample, written once and read once, at the least
        assert bytes_of[k] > 2 * 40 * 64 * 1920 * 1080
        assert bench.frame_traffic(k, 1920, 1080, 16) is None
        assert bench.frame_traffic(k, 640, 360, 64) is None
