"""The framework's work as timed cases, each through its public entry points.

The cases follow the stages a program built on the package runs: building
and refitting trees, skinning, tracing frames and ray buffers, the a-trous
and the learned denoiser, a training step, and a captured serving frame.
Sizes are those of the benchmark configurations (a 65,536-triangle cloud at
256 x 256, the 1.31 M-face mesh at 1080p, 500 k skinned vertices, 1080p
frames and 12 x 128 x 128 crops for the network), and small and odd ones
beside them. `listed` names the fixed cases, `draw` gives others of the same
ranges.
"""

from __future__ import annotations

import ctypes as C
import functools
import math

import numpy as np
import torch

import phiray_b200 as px
from phiray_b200 import scenes
from phiray_b200.batch import Batch
from phiray_b200.denoiser import Unet

# Face count of the displaced icosphere scene by subdivision level (with its
# two ground faces).
MESH_FACES = {lv: 20 * 4 ** lv + 2 for lv in range(3, 9)}
# Network layers: (input channels, output channels, level), in launch order.
LAYERS = [(16, 32, 0), (32, 32, 0), (32, 64, 1), (64, 64, 1), (64, 96, 2), (96, 96, 2), (96, 128, 3), (128, 128, 3),
          (128, 160, 4), (160, 160, 4), (288, 128, 3), (128, 128, 3), (224, 96, 2), (96, 96, 2), (160, 64, 1),
          (64, 64, 1), (96, 32, 0), (32, 32, 0), (32, 32, 0)]
# A late step of a decaying schedule: the weights barely move between passes.
LEARNING_RATE = 2e-6
ERR_WEIGHT = 0.1
THRESHOLD = 0.1


def listed() -> list[dict]:
    return [
        # the top tree over a scene's instances, or one small object: latency
        {"name": "lbvh_1k", "kind": "lbvh", "n": 1000},
        # a large mesh edited and rebuilt
        {"name": "lbvh_2m", "kind": "lbvh", "n": 2000000},
        # an animated mesh: new boxes, the same topology; an odd count
        {"name": "refit_1m", "kind": "refit", "n": 999001},
        # the tree the renderer walks by default, over a large mesh
        {"name": "sah_1m3", "kind": "sah", "n": 1310722},
        # posing a character's 500 k vertices
        {"name": "skin_500k", "kind": "skin", "n": 500000, "bones": 64},
        # a preview while samples still accumulate: the sums are kept
        {"name": "denoise_1080p", "kind": "denoise", "w": 1920, "h": 1080},
        # a small frame as a fresh tracer renders it: LBVH, the default kernel
        {"name": "render_cloud", "kind": "render", "scene": "cloud", "faces": 65536, "w": 256, "h": 256, "spp": 16,
         "bounces": 4, "tuned": False},
        # the whole frame of the large mesh: tree rebuilt, traced by the autotuned kernel, denoised
        {"name": "render_mesh_1080p", "kind": "render", "scene": "mesh", "level": 8, "w": 1920, "h": 1080, "spp": 16,
         "bounces": 8, "tuned": True},
        # incoherent rays from a caller's own buffer (baking, picking, ambient occlusion)
        {"name": "rays_bounce", "kind": "rays", "level": 8, "w": 1920, "h": 1080, "walk": 3},
        # the learned denoiser's network over one 1080p frame (padded to 1088 rows)
        {"name": "unet_1080p", "kind": "unet", "w": 1920, "h": 1080},
        # one step of training the denoiser
        {"name": "unet_train", "kind": "train", "batch": 12, "size": 128},
        # a serving frame: scenes rebuilt or refit, traced in one launch, denoised, as one graph
        {"name": "serve_6", "kind": "serve", "scenes": 6, "faces": 60000, "w": 512, "h": 512, "spp": 4},
    ]


def _log(rng, lo, hi) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    kind = rng.choice(["lbvh", "refit", "sah", "skin", "denoise", "render", "rays", "unet", "train", "serve"])
    if kind in ("lbvh", "refit"):
        return {"kind": kind, "n": _log(rng, 200, 2000000)}
    if kind == "sah":
        return {"kind": kind, "n": _log(rng, 500, 1310722)}
    if kind == "skin":
        return {"kind": kind, "n": _log(rng, 2000, 500000), "bones": rng.randint(8, 200)}
    if kind in ("denoise", "unet"):
        return {"kind": kind, "w": _log(rng, 100, 1920), "h": _log(rng, 100, 1080)}
    if kind == "train":
        return {"kind": kind, "batch": rng.randint(2, 12), "size": 16 * rng.randint(3, 8)}
    if kind == "rays":
        return {"kind": kind, "level": rng.randint(5, 8), "w": _log(rng, 60, 1920), "h": _log(rng, 60, 1080),
                "walk": rng.choice([0, 1, 3])}
    if kind == "serve":
        return {"kind": kind, "scenes": rng.randint(2, 6), "faces": _log(rng, 10000, 60000),
                "w": _log(rng, 100, 512), "h": _log(rng, 100, 512), "spp": rng.choice([1, 4])}
    case = {"kind": "render", "w": _log(rng, 120, 1920), "h": _log(rng, 90, 1080), "spp": rng.randint(1, 16),
            "bounces": rng.randint(2, 8), "tuned": rng.random() < 0.5}
    if rng.random() < 0.4:
        return {**case, "scene": "cloud", "faces": _log(rng, 2000, 65536), "w": min(case["w"], 640),
                "h": min(case["h"], 480)}
    return {**case, "scene": "mesh", "level": rng.randint(5, 8)}


# ---- what a program has in hand ----


@functools.cache
def _gpu() -> px.Gpu:
    """One context for the process, as a program keeps it."""
    return px.Gpu(0)


@functools.cache
def _base_scene(kind: str, size: int, width: int, height: int, spp: int, bounces: int):
    if kind == "cloud":
        return scenes.c1_plain(ntris=size, width=width, height=height, spp=spp, bounces=bounces)
    if kind == "mesh":
        return scenes.c2_mesh(levels=size, width=width, height=height, spp=spp, bounces=bounces)
    raise ValueError(kind)


@functools.cache
def _procedural(index: int, width: int, height: int, spp: int, faces: int):
    return scenes.procedural(index, width=width, height=height, spp=spp, bounces=6, target=faces)


def _turned(verts: np.ndarray, seed: int) -> np.ndarray:
    """The scene's vertices turned about the vertical axis by the seed's angle."""
    a = np.random.default_rng([seed, 11]).uniform(-0.4, 0.4)
    v = verts.copy()
    c, s = np.float32(math.cos(a)), np.float32(math.sin(a))
    v[:, 0], v[:, 2] = c * verts[:, 0] - s * verts[:, 2], s * verts[:, 0] + c * verts[:, 2]
    return v


def _generator(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(seed)


def _view(ptr: int, shape, typestr: str) -> torch.Tensor:
    """Device memory of the framework's as a tensor."""

    class _Memory:
        __cuda_array_interface__ = {"shape": tuple(shape), "typestr": typestr, "data": (ptr, False), "version": 3}

    return torch.as_tensor(_Memory(), device="cuda")


def _triangles(n: int, seed: int) -> torch.Tensor:
    """Small triangles with centroids uniform in the unit cube: (n, 3, 3)."""
    g = _generator(seed)

    def edge():
        d = torch.randn(n, 3, generator=g, device="cuda")
        return d / d.norm(dim=1, keepdim=True) * (0.005 + 0.015 * torch.rand(n, 1, generator=g, device="cuda"))

    c, e1, e2 = torch.rand(n, 3, generator=g, device="cuda"), edge(), edge()
    a = c - (e1 + e2) / 3.0
    return torch.stack([a, a + e1, a + e2], 1)


def _boxes(tri: torch.Tensor) -> torch.Tensor:
    """(n, 8) Aabb rows of the triangles."""
    out = torch.zeros(len(tri), 8, device=tri.device)
    out[:, 0:3], out[:, 4:7] = tri.amin(1), tri.amax(1)
    return out


def _planes(t: "px.Tracer") -> dict:
    """A tracer's image as its planes (a view: nothing is copied)."""
    n = t.w * t.h
    ptr, words = t.device_image()
    return _split(_view(ptr, (words,), "<i4"), n)


def _split(image: torch.Tensor, n: int) -> dict:
    f = image.view(torch.float32)
    return {"packed": image[:n], "sums": f[n:4 * n].view(n, 3).t(), "shown": f[4 * n:7 * n].view(n, 3).t(),
            "guides": f[7 * n:14 * n].view(n, 7).t(), "count": image[31 * n:32 * n]}


def _frame(w: int, h: int, seed: int, spp: int = 32) -> torch.Tensor:
    """A noisy traced image's px buffer: textured planes at several depths
    and a sky, `spp` samples a pixel, lone bright samples among them."""
    g = _generator(seed)
    n = w * h
    y, x = torch.meshgrid(torch.arange(h, device="cuda") / h, torch.arange(w, device="cuda") / w, indexing="ij")
    p = torch.rand(6, generator=g, device="cuda")
    region = (torch.floor(4 * x + 2 * p[0]) + 3 * torch.floor(3 * y + p[1])).long() % 7
    table = torch.rand(7, 8, generator=g, device="cuda")
    sky = (y < 0.15 + 0.1 * torch.sin(6 * x + 6 * p[2])).reshape(-1)
    alb = (0.1 + 0.8 * table[region][..., 0:3] * (0.7 + 0.3 * torch.sin(80 * x + 50 * y)[..., None])).reshape(n, 3)
    nrm = torch.nn.functional.normalize(table[region][..., 3:6] - 0.5, dim=-1).reshape(n, 3)
    depth = (1.0 + 4.0 * table[region][..., 6] + y).reshape(n)
    lit = (0.2 + table[region][..., 7] * (1.0 + torch.cos(5 * x - 3 * y)))[..., None].reshape(n, 1)
    noise = torch.rand(n, 3, generator=g, device="cuda") + torch.rand(n, 3, generator=g, device="cuda")
    spark = 1.0 + 30.0 * (torch.rand(n, 1, generator=g, device="cuda") < 0.001)
    light = alb * lit * noise * spark
    keep = (~sky).float()
    k = float(spp)
    image = torch.zeros(34 * n + 1, dtype=torch.int32, device="cuda")
    f = image.view(torch.float32)
    f[n:4 * n] = (light * keep[:, None] * k).reshape(-1)
    f[7 * n:10 * n] = (alb * keep[:, None] * k).reshape(-1)
    f[10 * n:13 * n] = (nrm * keep[:, None] * k).reshape(-1)
    f[13 * n:14 * n] = torch.where(sky, -torch.ones_like(depth), depth) * k
    f[24 * n:25 * n] = k
    image[31 * n:32 * n] = spp
    f[33 * n:34 * n] = sky.float() * k
    return image


def _features(B: int, Hp: int, Wp: int, h: int, w: int, seed: int) -> dict:
    """Network inputs of B noisy frames: features (bf16), irradiance and
    albedo planes, and a clean reference."""
    feat = torch.zeros(B, Hp, Wp, 16, device="cuda")
    irr, alb, ref = (torch.zeros(B, Hp, Wp, 3, device="cuda") for _ in range(3))
    for b in range(B):
        n = w * h
        f = _frame(w, h, seed + 1000 * b, 16).view(torch.float32)
        g = _generator(seed + 1000 * b + 1)
        k = 16.0
        sums, al = f[n:4 * n].reshape(h, w, 3), (f[7 * n:10 * n] / k).reshape(h, w, 3)
        met = torch.clamp(k - f[33 * n:34 * n].reshape(h, w, 1), min=1.0)
        ad = torch.clamp(al, min=0.05)
        ir = sums / met / ad
        d = (f[13 * n:14 * n] / k).reshape(h, w)
        x = feat[b, :h, :w]
        x[..., 0:3] = torch.log1p(0.25 * ir * torch.rand(h, w, 3, generator=g, device="cuda"))
        x[..., 3:6], x[..., 6:9] = torch.log1p(ir), al
        x[..., 9:12] = (f[10 * n:13 * n] / k).reshape(h, w, 3)
        x[..., 12], x[..., 13] = d / (1 + d.abs()), 1.0 - f[33 * n:34 * n].reshape(h, w) / k
        x[..., 14], x[..., 15] = 0.5, 1.0
        irr[b, :h, :w], alb[b, :h, :w] = ir, ad
        ref[b, :h, :w] = ad * torch.nn.functional.avg_pool2d(ir.permute(2, 0, 1)[None], 9, 1, 4)[0].permute(1, 2, 0)
    return {"feat": feat.to(torch.bfloat16), "irr": irr, "alb": alb, "ref": ref}


def _skin_inputs(case, seed):
    rng = np.random.default_rng([seed, 5])
    n, nb = case["n"], case["bones"]
    counts = rng.integers(1, 5, n)
    offsets = np.zeros(n + 1, np.uint32)
    offsets[1:] = np.cumsum(counts)
    k = int(offsets[-1])
    # neighbouring vertices hang on neighbouring bones
    near = (np.arange(n) * nb // n).repeat(counts)
    bone = np.clip(near + rng.integers(-2, 3, k), 0, nb - 1)
    pairs = np.zeros(k, scenes.PAIR)
    pairs["bone"], pairs["next"] = bone, np.clip(bone + 1, 0, nb - 1)
    pairs["blend"] = rng.random(k, dtype=np.float32)
    e = rng.exponential(1.0, k)
    pairs["weight"] = (e / np.add.reduceat(e, offsets[:-1].astype(np.int64)).repeat(counts)).astype(np.float32)
    rest = np.ones((n, 4), np.float32)
    rest[:, :3] = rng.uniform(-1.0, 1.0, (n, 3))
    m = np.zeros((nb, 4, 4), np.float32)
    for b in range(nb):
        axis = rng.standard_normal(3)
        m[b, :3, :3] = scenes._rot(axis, rng.uniform(-0.25, 0.25)).T
        m[b, 3, :3], m[b, 3, 3] = rng.uniform(-0.1, 0.1, 3), 1.0
    return rest, offsets, pairs, m.reshape(nb, 16)


def prepare(case, seed):
    gpu, kind = _gpu(), case["kind"]
    if kind in ("lbvh", "refit"):
        tri = _triangles(case["n"], seed)
        torch.cuda.synchronize()
        prims = _boxes(tri)
        torch.cuda.synchronize()
        s = {"case": case, "prims": prims, "bvh": px.GpuBvh.build_device(gpu, prims, case["n"], 4)}
        if kind == "refit":
            # the mesh in motion: every triangle drifts
            s["prims"] = _boxes(tri + 0.03 * torch.sin(7.0 * tri.flip(2)))
        n, d = case["n"], s["bvh"].device()
        s["out"] = _tree(_view(d["nodes"], (2 * n - 1, 8), "<f4"), _view(d["order"], (n,), "<i4"))
        torch.cuda.synchronize()
        return s
    if kind == "sah":
        n = case["n"]
        s = {"case": case, "prims": _boxes(_triangles(n, seed)), "nodes": torch.zeros(2 * n, 8, device="cuda"),
             "order": torch.zeros(n, dtype=torch.int32, device="cuda")}
        torch.cuda.synchronize()
        return s
    if kind == "skin":
        rest, offsets, pairs, bones = _skin_inputs(case, seed)
        dev = [torch.from_numpy(np.ascontiguousarray(a).view(np.uint8)).cuda() for a in (rest, offsets, pairs, bones)]
        s = {"case": case, "in": dev, "out": torch.empty(case["n"], 4, device="cuda")}
        torch.cuda.synchronize()
        return s
    if kind == "denoise":
        s = {"case": case, "px": _frame(case["w"], case["h"], seed)}
        torch.cuda.synchronize()
        return s
    if kind == "render":
        w, h = case["w"], case["h"]
        size = case["faces"] if case["scene"] == "cloud" else case["level"]
        base = _base_scene(case["scene"], size, w, h, case["spp"], case["bounces"])
        cam = px.camera(base)
        cam["w"], cam["h"] = w, h
        verts = _turned(base.verts, seed)
        t = px.Tracer(gpu, verts, base.faces, base.mats, normals=getattr(base, "normals", None))
        if case["tuned"]:
            t.set_tree(px.Tracer.TREE_SAH)
            t.autotune(cam, w, h, 1)
        s = {"case": case, "tracer": t, "cam": cam, "verts": torch.from_numpy(verts).cuda()}
        torch.cuda.synchronize()
        return s
    if kind == "rays":
        w, h = case["w"], case["h"]
        base = _base_scene("mesh", case["level"], w, h, 1, 8)
        cam = px.camera(base)
        cam["w"], cam["h"] = w, h
        t = px.Tracer(gpu, _turned(base.verts, seed), base.faces, base.mats)
        t.set_tree(px.Tracer.TREE_SAH)
        t.set_walk(case["walk"])
        rays = torch.empty(w * h, 8, device="cuda")
        t.secondary_rays(cam, w, h, seed % 4096, rays)
        s = {"case": case, "tracer": t, "rays": rays, "hits": torch.empty(w * h, 4, device="cuda")}
        torch.cuda.synchronize()
        return s
    if kind == "unet":
        w, h = case["w"], case["h"]
        Hp, Wp = (h + 15) // 16 * 16, (w + 15) // 16 * 16
        s = {"case": case, "net": Unet.pretrained(gpu), "size": (Hp, Wp), **_features(1, Hp, Wp, h, w, seed),
             "out": torch.empty(Hp, Wp, 3, device="cuda"), "err": torch.empty(Hp, Wp, device="cuda")}
        torch.cuda.synchronize()
        return s
    if kind == "train":
        B, z = case["batch"], case["size"]
        net = Unet.pretrained(gpu)
        s = {"case": case, "net": net, **_features(B, z, z, z, z, seed), "loss": torch.zeros(1, device="cuda"),
             "grads": net.grad_tensor().view(-1, 64).t(), "stream": torch.cuda.ExternalStream(gpu.stream)}
        torch.cuda.synchronize()
        return s
    # serve
    rng = np.random.default_rng([seed, 3])
    batch, tracers = Batch(gpu), []
    for k in range(case["scenes"]):
        faces = int(case["faces"] * 2.0 ** (k % 3 - 1))
        w, h = (case["w"], case["h"]) if k % 2 == 0 else (max(case["w"] // 2, 16), max(case["h"] // 2, 16))
        base = _procedural(200000 + k, w, h, case["spp"], faces)
        cam = px.camera(base)
        cam["w"], cam["h"] = w, h
        t = px.Tracer(gpu, _turned(base.verts, seed), base.faces, base.mats)
        tracers.append(t)
        batch.add(t, cam, w, h, 0, case["spp"])
    batch.autotune()
    net = Unet.pretrained(gpu)
    batch.capture(net, THRESHOLD)
    modes = rng.integers(0, 2, case["scenes"])
    torch.cuda.synchronize()
    return {"case": case, "batch": batch, "tracers": tracers, "net": net, "modes": modes}


# ---- one pass ----


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind in ("lbvh", "refit"):
        n, bvh = case["n"], s["bvh"]
        if kind == "lbvh":
            bvh.rebuild_device(s["prims"], n)
        else:
            bvh.update_device(s["prims"], n)
        return s["out"]
    if kind == "sah":
        lib, count, depth = px.lib(), C.c_uint32(), C.c_uint32()
        rc = lib.phx_bvh_build_sah(_gpu().handle, px.devptr(s["prims"]), case["n"], 4, px.devptr(s["nodes"]),
                                   px.devptr(s["order"]), C.byref(count), C.byref(depth))
        if rc < 0:
            raise px.PhxError(rc, "build_sah")
        return {**_tree(s["nodes"], s["order"]), "count": count.value, "depth": depth.value}
    if kind == "skin":
        rest, offsets, pairs, bones = s["in"]
        px.skin(_gpu(), rest, offsets, pairs, bones, case["bones"], s["out"], case["n"])
        return s["out"]
    if kind == "denoise":
        w, h = case["w"], case["h"]
        px.denoise(_gpu(), s["px"], w, h, keep=True)
        return {k: v for k, v in _split(s["px"], w * h).items() if k in ("packed", "shown")}
    if kind == "render":
        t, w, h = s["tracer"], case["w"], case["h"]
        t.repose_device(s["verts"], rebuild=True)
        t.trace(s["cam"], w, h, 0, case["spp"])
        if case["tuned"]:
            t.denoise()
        return _planes(t)
    if kind == "rays":
        s["tracer"].trace_rays(s["rays"], case["w"] * case["h"], s["hits"])
        hits = s["hits"]
        return {"t": hits[:, 0], "face": hits.view(torch.int32)[:, 1], "uv": hits[:, 2:4]}
    if kind == "unet":
        Hp, Wp = s["size"]
        s["net"].forward(s["feat"], s["irr"], s["alb"], 1, Hp, Wp, case["h"], case["w"], s["out"], s["err"])
        return {"out": s["out"], "err": s["err"]}
    if kind == "train":
        B, z = case["batch"], case["size"]
        with torch.cuda.stream(s["stream"]):
            s["loss"].zero_()
        s["net"].train_step(s["feat"], s["irr"], s["alb"], s["ref"], B, z, z, z, z, s["loss"], LEARNING_RATE,
                            ERR_WEIGHT)
        return {"grads": s["grads"], "loss": s["loss"]}
    s["batch"].replay(s["modes"])
    _, rays = s["batch"].results()
    # the float planes: what the readbacks of radiance and shown colour return
    images = [{k: v for k, v in _planes(t).items() if k in ("sums", "shown")} for t in s["tracers"]]
    return {"rays": rays.astype(np.int64), "images": images}


def _tree(nodes: torch.Tensor, order: torch.Tensor) -> dict:
    """A tree's arrays (views), its boxes and its index words apart."""
    return {"lo": nodes[:, 0:3], "hi": nodes[:, 4:7], "links": nodes.view(torch.int32)[:, 3::4], "order": order}


# ---- what one pass cannot do without ----


def work(case) -> dict:
    kind = case["kind"]
    if kind == "lbvh":
        return {"bytes": case["n"] * (32 + 64 + 4), "flops": 0}
    if kind == "refit":
        return {"bytes": case["n"] * (32 + 64 + 4), "flops": 0}
    if kind == "sah":
        return {"bytes": case["n"] * (32 + 32 + 4), "flops": 0}
    if kind == "skin":
        return {"bytes": case["n"] * (16 + 4 + 40 + 16), "flops": case["n"] * 2.5 * 80}
    if kind == "denoise":
        n = case["w"] * case["h"]
        return {"bytes": n * 4 * (3 + 3 + 3 + 1 + 4 + 3 + 4), "flops": n * 4 * 25 * 60}
    if kind == "render":
        faces = case["faces"] + 4 if case["scene"] == "cloud" else MESH_FACES[case["level"]]
        n = case["w"] * case["h"]
        # a path of some three rays a sample, about 20 node steps of 24 operations a ray
        return {"bytes": n * 4 * 26 + faces * (48 + 48), "flops": n * case["spp"] * 3.0 * 20 * 24}
    if kind == "rays":
        n = case["w"] * case["h"]
        return {"bytes": n * (32 + 16) + MESH_FACES[case["level"]] * 48, "flops": n * 20 * 24}
    if kind in ("unet", "train"):
        if kind == "unet":
            n = ((case["w"] + 15) // 16 * 16) * ((case["h"] + 15) // 16 * 16)
        else:
            n = case["batch"] * case["size"] ** 2
        flops = sum(2 * 9 * ci * co / 4 ** lv for ci, co, lv in LAYERS) * n
        params = sum(9 * ci * co + co for ci, co, _ in LAYERS)
        if kind == "unet":
            return {"bytes": n * (32 + 12 + 12 + 16) + params * 2, "flops": flops}
        return {"bytes": n * (32 + 12 + 12 + 12) + params * 4 * 7, "flops": 3 * flops}
    n = sum(case["w"] * case["h"] // (1 if k % 2 == 0 else 4) for k in range(case["scenes"]))
    net = sum(2 * 9 * ci * co / 4 ** lv for ci, co, lv in LAYERS)
    return {"bytes": n * 4 * 26 + case["scenes"] * case["faces"] * 96,
            "flops": n * (net + case["spp"] * 3.0 * 20 * 24)}


# ---- the same in 64 bits ----


def exact(case, seed):
    kind = case["kind"]
    if kind == "skin":
        rest, offsets, pairs, bones = _skin_inputs(case, seed)
        counts = np.diff(offsets.astype(np.int64))
        who = np.arange(case["n"]).repeat(counts)
        m = bones.astype(np.float64)
        b = pairs["blend"].astype(np.float64)[:, None]
        at = m[pairs["bone"]] + (m[pairs["next"]] - m[pairs["bone"]]) * b
        r = rest.astype(np.float64)[who]
        w = pairs["weight"].astype(np.float64)
        out = np.ones((case["n"], 4))
        total = np.bincount(who, w, case["n"])
        for j in range(3):
            p = at[:, j] * r[:, 0] + at[:, 4 + j] * r[:, 1] + at[:, 8 + j] * r[:, 2] + at[:, 12 + j]
            out[:, j] = np.bincount(who, w * p, case["n"]) / total
        return out
    if kind == "denoise":
        return {"packed": None, "shown": _denoise64(_frame(case["w"], case["h"], seed), case["w"], case["h"])}
    if kind == "unet":
        w, h = case["w"], case["h"]
        Hp, Wp = (h + 15) // 16 * 16, (w + 15) // 16 * 16
        x = _features(1, Hp, Wp, h, w, seed)
        with torch.no_grad():
            logits = _network64(_weights64(), x["feat"].double().permute(0, 3, 1, 2))
            out, err = _predict64(logits, x["irr"].double(), x["alb"].double(), h, w)
        full, e = torch.zeros(Hp, Wp, 3, dtype=torch.float64), torch.zeros(Hp, Wp, dtype=torch.float64)
        full[:h, :w], e[:h, :w] = out[0].cpu(), err[0].cpu()
        return {"out": full, "err": e}
    if kind == "train":
        return _train64(case, seed)
    return None


def _srgb64(c):
    c = c.clamp(0.0, 1.0)
    return torch.where(c <= 0.0031308, c * 12.92, 1.055 * c.pow(1.0 / 2.4) - 0.055)


def _denoise64(image, w, h):
    n = w * h
    f = image.view(torch.float32).double()
    k = 1.0 / image[31 * n:32 * n].clamp(min=1).double().reshape(h, w, 1)
    plane = lambda at, c: f[at * n:(at + c) * n].reshape(h, w, c)  # noqa: E731
    alb = _srgb64(plane(7, 3) * k)
    nrm = plane(10, 3) + 1e-9
    nrm = nrm / nrm.norm(dim=2, keepdim=True)
    depth = plane(13, 1) * k
    img = plane(1, 3) * k / alb.clamp(min=0.05)
    luma = torch.tensor([0.2126, 0.7152, 0.0722], dtype=torch.float64, device=image.device)
    rows, cols = torch.arange(h, device=image.device), torch.arange(w, device=image.device)

    def taps(dy, dx):
        ok = ((rows + dy >= 0) & (rows + dy < h))[:, None] & ((cols + dx >= 0) & (cols + dx < w))[None, :]
        at = ((rows + dy).clamp(0, h - 1)[:, None] * w + (cols + dx).clamp(0, w - 1)[None, :]).reshape(-1)
        return ok[..., None], lambda a: a.reshape(n, -1)[at].reshape(h, w, -1)

    for rnd, step in enumerate((1, 2, 4, 8)):
        centre = img
        if rnd == 0:
            top, total, met = torch.zeros_like(depth), torch.zeros_like(img), torch.zeros_like(depth)
            for dy in (-1, 0, 1):
                for dx in (-1, 0, 1):
                    if dy or dx:
                        ok, of = taps(dy, dx)
                        c = of(img) * ok
                        top, total, met = torch.maximum(top, (c @ luma)[..., None]), total + c, met + ok
            lone = (img @ luma)[..., None] > 1.5 * top + 0.05
            centre = torch.where(lone, total / met, img)
        lc = (centre @ luma)[..., None]
        total, weight = torch.zeros_like(img), torch.zeros_like(depth)
        for dy in range(-2, 3):
            for dx in range(-2, 3):
                ok, of = taps(dy * step, dx * step)
                tap = centre if dx == 0 and dy == 0 else of(img)
                jd = of(depth)
                ok = ok & ((jd < 0) == (depth < 0))
                dn = (1.0 - (nrm * of(nrm)).sum(2, keepdim=True)).clamp(min=0.0)
                da = (of(alb) - alb).norm(dim=2, keepdim=True)
                dd = (jd - depth).abs() / depth.abs().clamp(min=1e-3)
                dl = ((tap @ luma)[..., None] - lc).abs() / (0.08 + lc)
                kk = (0.375, 0.25, 0.0625)[abs(dx)] * (0.375, 0.25, 0.0625)[abs(dy)]
                wt = kk * torch.exp(-dn * 64.0 - da * 8.0 - dd * 40.0 - dl * dl * 7.0) * ok
                total, weight = total + tap * wt, weight + wt
        img = torch.where(weight > 0, total / weight, centre)
    met = 1.0 - plane(33, 1) * k
    lin = torch.where(met > 0.5 * k, img * alb.clamp(min=0.05), torch.zeros_like(img))
    shown = _srgb64((lin / torch.maximum(met, k)).clamp(min=0.0)).clamp(0.0, 1.0)
    return shown.reshape(n, 3).t().cpu()


def _weights64():
    """(W, b) of every layer from the shipped weights file: a 16-byte header,
    then per layer W [cout][3][3][cin] and b [cout] in float32."""
    raw = np.fromfile("phiray_b200/weights/kpcn.phxu", dtype="<f4", offset=16).astype(np.float64)
    out, at = [], 0
    for ci, co, _ in LAYERS:
        w = torch.from_numpy(raw[at:at + 9 * ci * co].reshape(co, 3, 3, ci)).permute(0, 3, 1, 2).cuda()
        at += 9 * ci * co
        out.append((w.contiguous(), torch.from_numpy(raw[at:at + co].copy()).cuda()))
        at += co
    return out


def _network64(params, x):
    conv = lambda i, v, relu=True: (torch.relu if relu else lambda q: q)(  # noqa: E731
        torch.nn.functional.conv2d(v, params[i][0], params[i][1], padding=1))
    skips = []
    for lv in range(4):
        x = conv(2 * lv + 1, conv(2 * lv, x))
        skips.append(x)
        x = torch.nn.functional.avg_pool2d(x, 2)
    x = conv(9, conv(8, x))
    for lv in (3, 2, 1, 0):
        x = torch.cat([torch.nn.functional.interpolate(x, scale_factor=2), skips.pop()], 1)
        at = 10 + 2 * (3 - lv)
        x = conv(at + 1, conv(at, x))
    return conv(18, x, False)


def _predict64(logits, irr, alb, h, w):
    wt = torch.softmax(logits[:, :25, :h, :w], 1)
    near = torch.nn.functional.pad(irr[:, :h, :w].permute(0, 3, 1, 2), (2, 2, 2, 2), mode="replicate")
    total = 0.0
    for t in range(25):
        total = total + wt[:, t:t + 1] * near[:, :, t // 5:t // 5 + h, t % 5:t % 5 + w]
    return alb[:, :h, :w] * total.permute(0, 2, 3, 1), (torch.exp(logits[:, 25, :h, :w]) - 1e-3).clamp(min=0.0)


def _train64(case, seed):
    B, z = case["batch"], case["size"]
    x = _features(B, z, z, z, z, seed)
    params = [(a.requires_grad_(), b.requires_grad_()) for a, b in _weights64()]
    logits = _network64(params, x["feat"].double().permute(0, 3, 1, 2))
    out, _ = _predict64(logits, x["irr"].double(), x["alb"].double(), z, z)
    ref = x["ref"].double()
    rel = (out - ref) ** 2 / (ref * ref + 0.01)
    target = torch.log(rel.mean(-1) + 1e-3).detach()
    (rel.mean() + ERR_WEIGHT * ((logits[:, 25] - target) ** 2).mean()).backward()
    flat = []
    for (ci, co, _), (a, b) in zip(LAYERS, params):
        rows = (9 * ci + 63) // 64 * 64
        g = torch.zeros(rows, co, dtype=torch.float64, device="cuda")
        g[:9 * ci] = a.grad.permute(2, 3, 1, 0).reshape(9 * ci, co)
        flat += [g.reshape(-1), b.grad]
    flat = torch.cat([torch.nn.functional.pad(v, (0, -len(v) % 64)) for v in flat])
    return {"grads": flat.view(-1, 64).t().cpu(), "loss": rel.mean().detach().reshape(1).cpu()}
