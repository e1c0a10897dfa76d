"""The renderer's workloads for performance measurements.

Each case is a dict of plain values; ``prepare`` makes what a program holds
before the call (a built and resident scene, output buffers, a prepared
batch), ``run`` makes one pass through the public API and returns what it
computed.  The sizes are those of the configurations in
``zigtrace_b200/scenes.py``, with small and odd ones beside them.

Kinds:
- ``render``: ``render_device`` of a resident scene into a device buffer, the
  call of a viewer or an animation loop (any scene family, either precision);
- ``render_host``: ``render`` into host memory;
- ``render_png``: ``render_png``, the command line's path from scene to file;
- ``batch``: a prepared ``Batch`` of many sphere fields, launched once;
- ``diff``: one optimisation step, ``forward`` and ``backward``;
- ``encode``: ``image_to_rgb8_device`` of a finished frame;
- ``png``: ``encode_png_device`` of an 8-bit frame;
- ``first_frame``: ``Scene.build(device=True)``, upload and a first small
  frame, what a program pays when its scene changes.
"""
from __future__ import annotations

import math
import struct
import zlib

import numpy as np
import torch

import zigtrace_b200 as zt
from zigtrace_b200 import scenes


# ------------------------------------------------------------------- cases --
def listed():
    return [
        # a viewer's preview while the camera moves: launch and latency count
        _render("preview_spheres", "render", "spheres", 18, 160, 90, 1, 16),
        # the command line's smallest job, an odd-sized thumbnail written as PNG
        _render("thumbnail_png", "render_png", "cornell", 0, 201, 113, 4, 16),
        # closed scene, long paths, few pixels (the Cornell configuration)
        _render("cornell", "render", "cornell", 0, 256, 256, 64, 16),
        # open scene of spheres, default precision (the random-spheres configuration)
        _render("spheres", "render", "spheres", 18, 1280, 720, 16, 50),
        # the same scene at an odd size into host memory, fast precision
        _render("spheres_fast_host", "render_host", "spheres", 18, 853, 479, 16, 50, fast=True),
        # the triangle-heavy configuration, fast precision: the headline frame
        _render("terrain_fast", "render", "terrain", 1000, 1920, 1080, 64, 16, fast=True),
        # a mid-size mesh at default precision, odd size
        _render("terrain", "render", "terrain", 500, 961, 541, 16, 16),
        # many small renders in one launch (the batched configuration)
        {"name": "batch_fields", "kind": "batch", "count": 256, "spp": 16, "max_depth": 16, "fast": True},
        # one step of an inverse-rendering loop (the differentiable configuration)
        {"name": "diff_step", "kind": "diff", "width": 512, "height": 512, "spp": 64, "max_depth": 16},
        # tone mapping and 8-bit encode of a full-HD frame
        {"name": "encode_1080p", "kind": "encode", "width": 1920, "height": 1080, "tonemap": "aces", "gamma": 2.2,
         "exposure": 1.0},
        # the PNG file of a full-HD frame
        {"name": "png_1080p", "kind": "png", "width": 1920, "height": 1080},
        # a new 1M-triangle scene: build, upload, first preview frame
        {"name": "first_frame", "kind": "first_frame", "size": 1000, "width": 160, "height": 90, "spp": 1,
         "max_depth": 16},
    ]


def _render(name, kind, family, size, width, height, spp, max_depth, fast=False):
    return {"name": name, "kind": kind, "family": family, "size": size, "width": width, "height": height, "spp": spp,
            "max_depth": max_depth, "fast": fast}


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["render", "render", "render", "render", "render_host", "render_png", "batch", "diff", "encode",
                       "png", "first_frame"])
    if kind in ("render", "render_host", "render_png"):
        family = rng.choice(["spheres", "terrain", "cornell"])
        # scene sizes: spheres on a grid of `size`, terrain cells along x
        size = {"spheres": lambda: _log(rng, 6, 40), "terrain": lambda: _log(rng, 60, 1000),
                "cornell": lambda: 0}[family]()
        width, height = _log(rng, 64, 1920), _log(rng, 36, 1080)
        # at most a quarter of the headline frame's samples, so that long paths cost no more than it
        spp = min(_log(rng, 1, 64), max(1, 33_000_000 // (width * height)))
        c = _render("", kind, family, size, width, height, spp, rng.choice([8, 16, 50]), rng.random() < 0.5)
        del c["name"]
        return c
    if kind == "batch":
        return {"kind": kind, "count": _log(rng, 8, 256), "spp": _log(rng, 2, 16), "max_depth": rng.choice([8, 16]),
                "fast": rng.random() < 0.5}
    if kind == "diff":
        return {"kind": kind, "width": _log(rng, 48, 512), "height": _log(rng, 48, 512), "spp": _log(rng, 4, 64),
                "max_depth": rng.choice([8, 16])}
    if kind == "encode":
        return {"kind": kind, "width": _log(rng, 64, 3840), "height": _log(rng, 36, 2160),
                "tonemap": rng.choice(["none", "reinhard", "aces"]), "gamma": rng.choice([1.0, 1.8, 2.2, 2.4]),
                "exposure": round(rng.uniform(0.25, 4.0), 3)}
    if kind == "png":
        return {"kind": kind, "width": _log(rng, 16, 3840), "height": _log(rng, 9, 2160)}
    return {"kind": kind, "size": _log(rng, 60, 1000), "width": _log(rng, 64, 320), "height": _log(rng, 36, 180),
            "spp": 1, "max_depth": 16}


# ----------------------------------------------------------------- prepare --
def _scene(family, size, seed):
    if family == "spheres":
        return scenes.random_spheres(seed, grid=size)
    if family == "terrain":
        return scenes.triangle_heavy(seed, nx=size, nz=max(size // 2, 1))
    # the Cornell box with its two objects' materials and light from the seed
    rng = np.random.default_rng(seed)
    s = scenes.cornell(float(rng.choice([0.0, rng.uniform(0.0, 0.3)])))
    colors = s.materials["color"].copy()
    colors[:3] *= rng.uniform(0.8, 1.2, (3, 3))
    colors[3] *= rng.uniform(0.8, 1.2)
    return zt.set_colors(s, colors)


def _options(case, seed):
    return zt.Options(width=case["width"], height=case["height"], spp=case["spp"], max_depth=case["max_depth"],
                      seed=seed)


def _config(case):
    return zt.GpuConfig(precision=zt.PRECISION_FAST) if case["fast"] else None


def _frame(case, seed):
    """An HDR frame's values: mostly within the displayable range, some
    highlights and black."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = case["width"] * case["height"] * 3
    v = torch.rand(n, generator=g, device="cuda", dtype=torch.float64)
    v = v * v * 4.0
    v[torch.rand(n, generator=g, device="cuda") < 0.05] = 0.0
    return v


def _pointer(t):
    return t.data_ptr(), torch.cuda.current_stream().cuda_stream


def prepare(case, seed):
    kind = case["kind"]
    n = case.get("width", 0) * case.get("height", 0)
    state = {"case": case}
    if kind in ("render", "render_host", "render_png"):
        state["scene"] = _scene(case["family"], case["size"], seed).build(device=True)
        state["scene"].upload()
        state["options"], state["config"] = _options(case, seed), _config(case)
        if kind == "render":
            state["out"] = torch.empty((n, 3), dtype=torch.float64, device="cuda")
    elif kind == "batch":
        # the workload's sphere counts (log-uniform) and resolutions; the fields
        # themselves and the streams from the seed
        rng = np.random.default_rng(case["count"])
        work = []
        for k in range(case["count"]):
            spheres = int(math.exp(rng.uniform(math.log(16), math.log(20000))))
            w, h = scenes.BATCH_RESOLUTIONS[int(rng.integers(len(scenes.BATCH_RESOLUTIONS)))]
            work.append((scenes.sphere_field(seed + k, spheres).build(),
                         zt.Options(width=w, height=h, spp=case["spp"], max_depth=case["max_depth"], seed=seed + k)))
        sizes = [o.width * o.height * 3 for _, o in work]
        state["out"] = torch.empty(sum(sizes), dtype=torch.float64, device="cuda")
        starts = np.concatenate([[0], np.cumsum(sizes)[:-1]])
        state["batch"] = zt.Batch([s for s, _ in work], [o for _, o in work],
                                  [state["out"].data_ptr() + 8 * int(a) for a in starts], _config(case))
    elif kind == "diff":
        scene, target = scenes.cornell_diff(seed)
        scene.build()
        scene.upload()
        rng = np.random.default_rng(seed)
        state["scene"], state["options"] = scene, _options(case, seed)
        state["colors"] = scene.materials["color"] * rng.uniform(0.9, 1.1, target.shape)
        photo = zt.Options(width=case["width"], height=case["height"], spp=2, max_depth=case["max_depth"],
                           seed=seed + 1)
        state["target"] = zt.forward(scene, photo, target).pixels
    elif kind == "encode":
        state["pixels"] = _frame(case, seed)
        state["out"] = torch.empty(3 * n, dtype=torch.uint8, device="cuda")
        state["output"] = zt.Output(case["tonemap"], case["gamma"], case["exposure"])
    elif kind == "png":
        state["rgb"] = (_frame(case, seed).clamp(0.0, 1.0) * 255.0).round().to(torch.uint8)
        state["size"] = zt.png_size(case["width"], case["height"])
        state["out"] = torch.empty(state["size"], dtype=torch.uint8, device="cuda")
    elif kind == "first_frame":
        state["scene"] = _scene("terrain", case["size"], seed)
        state["options"] = _options(case, seed)
    return state


# --------------------------------------------------------------------- run --
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "render":
        out, stream = _pointer(state["out"])
        zt.render_device(state["scene"], state["options"], out, stream, state["config"])
        return state["out"]
    if kind == "render_host":
        return zt.render(state["scene"], state["options"], state["config"]).pixels
    if kind == "render_png":
        return np.frombuffer(zt.render_png(state["scene"], state["options"], zt.Output(tonemap="aces"),
                                           state["config"]), np.uint8)
    if kind == "batch":
        state["batch"].launch(torch.cuda.current_stream().cuda_stream)
        return state["out"]
    if kind == "diff":
        image = zt.forward(state["scene"], state["options"], state["colors"]).pixels
        d_image = (image - state["target"]) * (2.0 / image.size)
        return {"image": image, "gradient": zt.backward(state["scene"], state["options"], d_image, state["colors"])}
    if kind == "encode":
        out, stream = _pointer(state["out"])
        zt.image_to_rgb8_device(state["pixels"].data_ptr(), case["width"] * case["height"], out, state["output"],
                                stream)
        return state["out"]
    if kind == "png":
        out, stream = _pointer(state["out"])
        zt.encode_png_device(state["rgb"].data_ptr(), case["width"], case["height"], out, state["size"], stream)
        return state["out"]
    scene = state["scene"].build(device=True)
    return zt.render(scene, state["options"]).pixels


# -------------------------------------------------------------------- work --
# Rays per sample and shaded hits per sample of the families, counted on the
# CPU at the configurations' sizes.
_RAYS = {"cornell": (5.4, 3.0), "spheres": (2.4, 1.5), "terrain": (1.9, 0.6)}


def _trace_work(family, prims, samples, pixels):
    """Least work of a render: a root-to-leaf descent (two box tests a level,
    12 operations each) and two primitive tests (40) per ray, 170 operations
    per shaded hit and camera ray; the scene (80 bytes a primitive) read and
    the frame (24 bytes a pixel) written once."""
    rays, hits = _RAYS[family]
    per_sample = rays * (24.0 * math.log2(max(prims, 2)) + 80.0) + 170.0 * (hits + 1.0)
    return 80.0 * prims + 24.0 * pixels, per_sample * samples


def work(case):
    kind = case["kind"]
    n = case.get("width", 0) * case.get("height", 0)
    if kind in ("render", "render_host", "render_png"):
        prims = {"cornell": 14, "spheres": case["size"] ** 2, "terrain": case["size"] ** 2 + 25_728}[case["family"]]
        b, f = _trace_work(case["family"], prims, n * case["spp"], n)
        return {"bytes": b, "flops": f}
    if kind == "batch":  # mean of the workload's resolutions and sphere counts
        pixels = case["count"] * 58_368
        b, f = _trace_work("spheres", 2_800, pixels * case["spp"], pixels)
        return {"bytes": b + 80.0 * 2_800 * (case["count"] - 1), "flops": f}
    if kind == "diff":  # the image and its gradient: two walks of every path
        b, f = _trace_work("cornell", 64, n * case["spp"], 2 * n)
        return {"bytes": b, "flops": 2.0 * f}
    if kind == "encode":
        return {"bytes": 27.0 * n, "flops": 60.0 * n}
    if kind == "png":
        return {"bytes": 3.0 * n + zt.png_size(case["width"], case["height"]), "flops": 0.0}
    prims = case["size"] ** 2 + 25_728
    levels = math.log2(prims)
    # shapes read, a node pair and a primitive record written; 3 axes binned on every level
    return {"bytes": (80.0 + 112.0 + 80.0) * prims, "flops": 30.0 * prims * levels}


# ------------------------------------------------------------------- exact --
def exact(case, seed):
    """The bytes of the output stage in plain NumPy and zlib.  A rendered image
    has no such value: it is defined by its random streams path by path."""
    state = prepare(case, seed) if case["kind"] in ("encode", "png") else None
    if case["kind"] == "encode":
        x = np.maximum(state["pixels"].cpu().numpy() * case["exposure"], 0.0)
        if case["tonemap"] == "reinhard":
            x = x / (1.0 + x)
        elif case["tonemap"] == "aces":
            x = (x * (2.51 * x + 0.03)) / (x * (2.43 * x + 0.59) + 0.14)
        x = np.clip(x, 0.0, 1.0) ** (1.0 / case["gamma"])
        return np.floor(np.clip(x, 0.0, 1.0) * 255.0 + 0.5).astype(np.uint8)
    if case["kind"] == "png":
        w, h = case["width"], case["height"]
        rows = np.zeros((h, 3 * w + 1), np.uint8)
        rows[:, 1:] = state["rgb"].cpu().numpy().reshape(h, 3 * w)
        raw = rows.tobytes()
        data = b"\x78\x01"
        for a in range(0, len(raw), 65535):
            part = raw[a:a + 65535]
            data += struct.pack("<BHH", a + 65535 >= len(raw), len(part), len(part) ^ 0xFFFF) + part
        data += struct.pack(">I", zlib.adler32(raw))

        def chunk(name, body):
            return struct.pack(">I", len(body)) + name + body + struct.pack(">I", zlib.crc32(name + body))

        return np.frombuffer(b"\x89PNG\r\n\x1a\n" + chunk(b"IHDR", struct.pack(">IIBBBBB", w, h, 8, 2, 0, 0, 0)) +
                             chunk(b"IDAT", data) + chunk(b"IEND", b""), np.uint8)
    return None
