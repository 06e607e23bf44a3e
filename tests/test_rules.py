"""The host's decisions between paths (phiray_b200/csrc/rules.cuh), built for
the host: which calls take which path, over the forms that they accept."""

import ctypes as C
import subprocess
from pathlib import Path

import pytest

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
