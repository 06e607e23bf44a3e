"""The subtree kernels of the device's SAH build, a warp's lanes run as threads
of the host, against the oracle's restatement of Bvh::build_sah: nodes, bounds,
slot order and depth, word for word."""

import ctypes as C
import subprocess
from pathlib import Path

import numpy as np
import pytest

HERE = Path(__file__).resolve().parent


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = tmp_path_factory.mktemp("sahwarp") / "libsahwarp.so"
    subprocess.run(["g++", "-O1", "-std=c++20", "-pthread", "-shared", "-fPIC", "-ffp-contract=off", "-fno-fast-math",
                    "-Wno-unknown-pragmas", "-o", str(out), str(HERE / "sah_warp.cpp")], check=True)
    return C.CDLL(str(out))


@pytest.fixture(scope="module")
def build(lib):
    lib.warp_build_sah.restype = C.c_uint32

    def run(prims, leaf, vec):
        n = len(prims)
        raw = np.zeros(8 * n + 4, np.float32)  # a 16-byte boundary for the wide accesses, one word past it else
        at = (-raw.ctypes.data // 4) % 4 + (0 if vec else 1)
        p = raw[at: at + 8 * n]
        p[:] = prims.reshape(-1)
        nodes, order, depth = np.zeros((2 * n, 8), np.float32), np.zeros(n, np.uint32), C.c_uint32()
        m = lib.warp_build_sah(C.c_void_p(p.ctypes.data), n, leaf, int(vec), C.c_void_p(nodes.ctypes.data),
                               C.c_void_p(order.ctypes.data), C.byref(depth))
        return nodes[:m], order, depth.value

    return run


def _boxes(n, kind):
    rng = np.random.default_rng(n)
    p = np.zeros((n, 8), np.float32)
    lo = rng.uniform(-1.0, 1.0, (n, 3)).astype(np.float32)
    if kind == "grid":  # many equal costs and shared bins
        lo = np.round(lo * 2.0) / 2.0
    elif kind == "outliers":  # splits of a few slots against the rest, at many scales
        lo *= np.exp(-rng.uniform(0.0, 12.0, (n, 1))).astype(np.float32)
    elif kind == "nan":  # bounds that are not numbers lose
        lo[::5, 1] = np.nan
    elif kind == "inf":  # areas and costs that are not finite
        lo[::7, 0] = np.inf
        lo[::3, 2] = -np.inf
    elif kind == "inverted":  # high corners below the low ones
        p[:, 4:7] = lo - 0.3
    p[:, 0:3] = lo
    if kind != "inverted":
        with np.errstate(invalid="ignore"):
            p[:, 4:7] = lo + rng.uniform(0.0, 0.1, (n, 3)).astype(np.float32)
    return p


@pytest.mark.parametrize("n,leaf,vec", [(1, 1, True), (2, 1, False), (31, 4, True), (33, 1, False), (64, 2, True),
                                        (127, 1, True), (127, 200, True)])
@pytest.mark.parametrize("kind", ["plain", "grid", "outliers", "nan", "inf", "inverted"])
def test_a_warps_subtree_is_the_reference_tree(build, orc, n, leaf, vec, kind):
    p = _boxes(n, kind)
    want_nodes, want_order, want_depth = orc.build_sah(p, leaf)
    nodes, order, depth = build(p, leaf, vec)
    assert depth == want_depth
    assert np.array_equal(order, want_order)
    assert np.array_equal(nodes.view(np.uint32), want_nodes.view(np.uint32))


@pytest.mark.parametrize("n", [1, 127, 128, 129, 300, 5000, 100_000])
@pytest.mark.parametrize("cut", ["one", "half", "seed", "mixed"])
def test_open_nodes_bounds_what_a_build_opens(lib, n, cut):
    """Nodes opened by the build's rule (128 slots or more, up to depth 30)
    when every node parts as unevenly, evenly or awkwardly as it can."""
    rng = np.random.default_rng(n)
    opened, level = 1, [n]
    for _ in range(31):
        children = []
        for k in level:
            if k < 128:
                continue
            kind = cut if cut != "mixed" else ("one", "half", "seed")[rng.integers(3)]
            m = {"one": 1, "half": k // 2, "seed": min(127, k - 1)}[kind]
            children += [m, k - m]
        opened += len(children)
        level = children
    assert opened <= lib.warp_open_nodes(n) <= 2 * n - 1
