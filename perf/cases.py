"""Performance cases: the work a user of this library has it do, through its
public entry points (include/arbor.h by way of arbor_b200).

Kinds of case:

  scene     arbor_buildScene: grow a tree, its records, Morton order and BVH
            (a new seed, the rebuild of an animated scene every frame, or the
            scenes of a forest of several species back to back)
  frame     one rendered image: per sample arbor_setSample, tracePixels,
            shadePixels, filterResolve on one resident scene (the forest of
            324 trees, the single tree, or a forest of several species), with
            or without sun shadows and wind, optionally rebuilding the scene
  batch     arbor_batch_*: many views of many scenes, one graph launch, the
            pixels read back to the host
  filter    arbor_filterResolve alone on a large image with history
  denoise   the learned denoiser on one frame: filterLighting, features, the
            network
  train     forward and backward of the denoiser on a batch of crops
            (arbor_denoiser_gradient)

Rendered outputs have no 64-bit value to compare with: which primitive a ray
hits is a discrete decision of the FP32 solve (a 64-bit rerun of the same
formulas moves about 3 % of the hit ids), so `exact` gives None for them, as
for keys, orders and bytes.  The filter and the network have one.
"""
from __future__ import annotations

import ctypes
import math
import os
import sys

import numpy as np
import torch

_PACKAGE = os.path.abspath("arbor-cuda_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(0, _PACKAGE)

import arbor_b200 as ab  # noqa: E402
import workloads  # noqa: E402

FAR = 100000.0
SEEDS = workloads.batch_seeds(16)  # the 16 master seeds of the batched workload
# (cin, cout, leaky ReLU) of the denoiser's convolutions (include/arbor.h: 32/64/96/128 channels, 3x3)
LAYERS = ((16, 32, 1), (32, 32, 1), (32, 64, 1), (64, 64, 1), (64, 96, 1), (96, 96, 1), (96, 128, 1), (128, 128, 1), (224, 96, 1),
          (96, 96, 1), (160, 64, 1), (64, 64, 1), (96, 32, 1), (32, 32, 1), (32, 16, 0))
LEVEL = (0, 0, 1, 1, 2, 2, 3, 3, 2, 2, 1, 1, 0, 0, 0)
MACS = sum(9.0 * cin * (3 if k == 14 else cout) / 4 ** LEVEL[k] for k, (cin, cout, _) in enumerate(LAYERS))  # per pixel
SCENE_BYTES = 4.0 * (32768 * 24 + 65536 * 8 + 32768)  # P, Nodes, Order


def listed() -> list[dict]:
    return [
        # The smallest call: a scene build, a few launches of latency each.
        {"name": "scene_build", "kind": "scene", "scenes": 1},
        # One tree, 256 x 256, shadows off: the smallest measured rendering configuration.
        {"name": "tree_256", "kind": "frame", "scene": "tree", "width": 256, "height": 256, "spp": 1, "shadows": False, "wind": 0.0},
        # A small window of odd size, sun shadows on.
        {"name": "forest_333x187", "kind": "frame", "scene": "forest", "width": 333, "height": 187, "spp": 1, "shadows": True, "wind": 0.0},
        # The headline frame: the forest at full HD, shadows off ...
        {"name": "forest_1080p", "kind": "frame", "scene": "forest", "width": 1920, "height": 1080, "spp": 1, "shadows": False, "wind": 0.0},
        # ... and with tree-to-tree sun shadows.
        {"name": "forest_sun_1080p", "kind": "frame", "scene": "forest", "width": 1920, "height": 1080, "spp": 1, "shadows": True, "wind": 0.0},
        # Progressive samples of an animated frame: wind, shadows, the scene rebuilt.
        {"name": "wind_4spp_540p", "kind": "frame", "scene": "forest", "width": 960, "height": 540, "spp": 4, "shadows": True, "wind": 0.6,
         "rebuild": True},
        # A forest of 16 species (16 resident scenes).
        {"name": "species_720p", "kind": "frame", "scene": "species", "species": 16, "width": 1280, "height": 720, "spp": 1, "shadows": True,
         "wind": 0.0},
        # Offline rendering of many views of mixed size, pixels back to the host.
        {"name": "batch_16_views", "kind": "batch", "views": 16, "scenes": 4, "largest": 1920 * 1080, "shadows": True},
        # Filter and resolve of an ultra-HD progressive frame.
        {"name": "filter_2160p", "kind": "filter", "width": 3840, "height": 2160, "sample": 3},
        # The learned denoiser on a small and a full-HD frame.
        {"name": "denoise_360p", "kind": "denoise", "width": 640, "height": 360},
        {"name": "denoise_1080p", "kind": "denoise", "width": 1920, "height": 1080},
        # Its training at the batch and crop of the training recipe.
        {"name": "train_4x256", "kind": "train", "batch": 4, "width": 256, "height": 256},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng) -> dict:
    kind = rng.choice(("scene", "frame", "frame", "frame", "frame", "frame", "batch", "filter", "denoise", "denoise", "train"))
    if kind == "scene":
        return {"kind": "scene", "scenes": _log_int(rng, 1, 64)}
    if kind == "frame":
        scene = rng.choice(("tree", "forest", "forest", "forest", "species"))
        height = _log_int(rng, 96, 1080)
        width = min(1920, max(64, int(height * rng.uniform(0.9, 1.9))))
        case = {"kind": "frame", "scene": scene, "width": width, "height": height, "spp": 1, "shadows": rng.random() < 0.6,
                "wind": rng.choice((0.0, 0.0, 0.6))}
        if scene == "species":
            case["species"] = _log_int(rng, 2, 16)
        elif width * height <= 960 * 540:
            case["spp"] = rng.choice((1, 2, 4))
            case["rebuild"] = rng.random() < 0.3
        return case
    if kind == "batch":
        return {"kind": "batch", "views": _log_int(rng, 2, 16), "scenes": rng.randint(1, 4), "largest": rng.choice((640 * 360, 1280 * 720)),
                "shadows": rng.random() < 0.6}
    if kind == "filter":
        height = _log_int(rng, 64, 2160)
        return {"kind": "filter", "width": max(32, int(height * rng.uniform(0.8, 1.77))), "height": height, "sample": rng.choice((0, 1, 3, 15))}
    if kind == "denoise":
        height = 8 * _log_int(rng, 8, 135)
        return {"kind": "denoise", "width": min(1920, 8 * max(8, int(height * rng.uniform(0.9, 1.78) / 8))), "height": height}
    size = 8 * rng.randint(8, 32)
    return {"kind": "train", "batch": rng.randint(1, 4), "width": size, "height": 8 * rng.randint(8, 32)}


# ------------------------------------------------------------------ inputs --
def _check(status: int) -> None:
    ab.check(status)


def _f(n: int) -> torch.Tensor:
    return torch.zeros(n, dtype=torch.float32, device="cuda")


def _i(n: int) -> torch.Tensor:
    return torch.zeros(n, dtype=torch.int32, device="cuda")


def _pick(seed: int) -> int:
    return SEEDS[seed % len(SEEDS)]


class _Scene:
    """n scenes back to back (one, or one per species)."""

    def __init__(self, seeds: list[int]):
        n = len(seeds)
        self.seeds = seeds
        self.B, self.P, self.Nodes = _f(2109 * 20), _f(n * 32768 * 24), _f(n * 65536 * 8)
        self.Keys, self.Order, self.scratch = _i(32768), _i(n * 32768), _i(2 * 32768)
        self.C = _f(64)
        for k in range(n):
            self.build(k)

    def build(self, k: int = 0) -> None:
        _check(ab.call("arbor_buildScene", self.seeds[k], self.B, self.P[k * 32768 * 24:], self.Keys, self.Order[k * 32768:],
                       self.Nodes[k * 65536 * 8:], self.C, self.scratch))


def _state(case: dict, seed: int, scene_seed: int) -> np.ndarray:
    """Camera record of a seeded first-person pose."""
    r = [workloads.rnd(k, 7919 * seed + 13) for k in range(5)]
    w, h = case["width"], case["height"]
    if case["scene"] == "tree":
        C = workloads.single_tree_camera(w, h, scene_seed)
        angle = 2.0 * math.pi * r[0]
        C[0], C[2] = 6.0 * math.sin(angle), 6.0 * math.cos(angle)
        if case["shadows"]:
            C[22] = 1.0
            C[12], C[13] = workloads.shadow_sun(scene_seed)
    else:
        C = workloads.view_pose_state(scene_seed, w, h, (2.0 * r[0] - 1.0) * 200.0, (2.0 * r[1] - 1.0) * 200.0, 2.0 * math.pi * r[2],
                                      -0.05 + 0.25 * r[3], case["shadows"])
    C[11] = case["wind"]
    C[8] = 8.0 * r[4] if case["wind"] else 0.0
    return C


class _Frame:
    def __init__(self, case: dict, seed: int):
        self.case = case
        n = case.get("species", 1)
        first = seed % len(SEEDS)
        seeds = [SEEDS[(first + k) % len(SEEDS)] for k in range(n)]
        self.scene = _Scene(seeds)
        self.C = torch.from_numpy(_state(case, seed, seeds[0])).cuda()  # the camera; scene.C is the builds' default one
        px = case["width"] * case["height"]
        self.Hit, self.Linear, self.Guide, self.Filtered, self.History = (_f(4 * px) for _ in range(5))
        self.Pixels = _i(px)
        if case["scene"] == "species":
            self.of = (ctypes.c_int * 324)(*[int(x) for x in workloads.species_of(n, seeds[0])])

    def run(self):
        c, s = self.case, self.scene
        w, h = c["width"], c["height"]
        if c.get("rebuild"):
            s.build()
        for k in range(c["spp"]):
            _check(ab.call("arbor_setSample", self.C, k, int(k == 0)))
            if c["scene"] == "species":
                _check(ab.call("arbor_traceSpeciesPixels", s.P, s.Nodes, s.Order, c["species"], self.of, self.C, self.Hit, w, h))
                _check(ab.call("arbor_shadeSpeciesPixels", s.P, s.Nodes, s.Order, c["species"], self.of, self.C, self.Hit, self.Linear,
                               self.Guide, w, h))
            else:
                form = "Tree" if c["scene"] == "tree" else ""
                _check(ab.call(f"arbor_trace{form}Pixels", s.P, s.Nodes, s.Order, self.C, self.Hit, w, h))
                _check(ab.call(f"arbor_shade{form}Pixels", s.P, s.Nodes, s.Order, self.C, self.Hit, self.Linear, self.Guide, w, h))
            _check(ab.call("arbor_filterResolve", self.Linear, self.Guide, self.Hit, self.Filtered, self.History, self.Pixels, self.C, w, h))
        return {"Hit": self.Hit, "Linear": self.Linear, "Guide": self.Guide, "Filtered": self.Filtered, "History": self.History,
                "Pixels": self.Pixels}


class _Build(_Scene):
    def __init__(self, case: dict, seed: int):
        super().__init__([_pick(seed + k) for k in range(case["scenes"])])

    def run(self):
        for k in range(len(self.seeds)):
            self.build(k)
        return {"P": self.P, "Order": self.Order, "Nodes": self.Nodes, "Keys": self.Keys, "C": self.C}


class _Batch:
    """The loop of a batch job: cameras up, one render, pixels back."""

    def __init__(self, case: dict, seed: int):
        first = seed % len(SEEDS)
        seeds = [SEEDS[(first + k) % len(SEEDS)] for k in range(case["scenes"])]
        sizes = [r for r in workloads.BATCH_RESOLUTIONS if r[0] * r[1] <= case["largest"]]
        # the mix of sizes is the case's own (each size in turn), the poses the seed's
        poses = workloads.batch_views(case["views"], seeds, resolutions=sizes[:1], seed=1000 + seed, shadows=case["shadows"])
        views = []
        for k, (scene, _, _, C) in enumerate(poses):
            w, h = sizes[k % len(sizes)]
            C = C.copy()
            C[32], C[33] = w, h
            views.append((scene, w, h, C))
        self.cameras = np.stack([v[3] for v in views])
        self.batch = ab.Batch(seeds, views)
        self.pixels = torch.empty(sum(v[1] * v[2] for v in views), dtype=torch.int32, pin_memory=True)

    def run(self):
        self.batch.set_cameras(self.cameras)
        self.batch.render()
        self.batch.read_pixels_into(self.pixels.data_ptr(), self.pixels.numel())
        return self.pixels


def _gbuffer(n: int, width: int, height: int, seed: int) -> dict[str, torch.Tensor]:
    """n images of a forest-like G-buffer: sky above a ragged skyline, ground,
    and surfaces (primitive and tree ids) in patches of a few pixels, depths
    of 1.5-120 m smooth inside a patch, radiance = albedo x light with the
    1-spp light of a sun that is visible in part of the samples.  (n, h, w, .)"""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    g = torch.Generator(device=dev).manual_seed(seed)
    u = lambda *s: torch.rand(*s, generator=g, device=dev)  # noqa: E731
    y = torch.arange(height, device=dev).view(1, height, 1).expand(n, height, width)
    x = torch.arange(width, device=dev).view(1, 1, width).expand(n, height, width)
    # ragged patches: cells of 8 x 6 pixels whose borders are jittered by a hash of the position
    jx, jy = (u(n, height, width) * 3.0).long(), (u(n, height, width) * 3.0).long()
    cw, ch = width // 8 + 3, height // 6 + 3
    cell = (torch.arange(n, device=dev).view(n, 1, 1) * ch + (y + jy) // 6) * cw + (x + jx) // 8
    cells = n * ch * cw
    prim = (u(cells) * 29412).floor()
    tree = (u(cells) * 324).floor()
    base = 1.5 * torch.exp(u(cells) * math.log(80.0))
    skyline = (0.35 + 0.2 * u(n, 1, width)) * height
    skyline = torch.nn.functional.avg_pool1d(skyline, 9, 1, 4, count_include_pad=False).view(n, 1, width)
    is_sky = (y < skyline) & (u(cells)[cell] < 0.55)
    is_ground = (~is_sky) & (y > 0.8 * height)
    t = base[cell] * (1.0 + 0.002 * u(n, height, width))
    t = torch.where(is_ground, 1.72 * height / (y + 1.0 - 0.45 * height).clamp(min=1.0), t)
    t = torch.where(is_sky, torch.full_like(t, FAR), t)
    none = torch.full_like(t, -1.0)
    hit = torch.stack([t, torch.where(is_sky | is_ground, none, prim[cell]), torch.where(is_sky | is_ground, none, tree[cell]),
                       0.9 * t / height], -1).float()
    albedo = (0.04 + 0.3 * u(cells, 3))[cell] * (0.9 + 0.2 * u(n, height, width, 1))
    albedo = torch.where(is_sky[..., None], torch.ones_like(albedo), albedo)
    light = torch.where(u(n, height, width, 1) < 0.4, 0.15 + 4.0 * u(n, height, width, 1), 0.25 + 0.1 * u(n, height, width, 1))
    light = torch.where(is_sky[..., None], 0.3 + 0.5 * u(n, height, 1, 1).expand_as(light), light)
    one = torch.ones(n, height, width, 1, device=dev)
    normal = torch.nn.functional.normalize((u(cells, 3) - 0.5)[cell] + torch.tensor([0.0, 0.4, 0.0], device=dev), dim=-1)
    normal = torch.where(is_sky[..., None], torch.zeros_like(normal), normal)
    cat = lambda v, w: torch.cat([v, w], -1).float().contiguous()  # noqa: E731
    return {"Hit": hit.contiguous(), "Guide": cat(albedo, one), "Linear": cat(albedo * light, one), "Normal": cat(normal, 0.0 * one),
            "Mean": cat(albedo * torch.where(is_sky[..., None], light, 0.25 + 0.75 * torch.ones_like(light)), one)}


class _Filter:
    def __init__(self, case: dict, seed: int):
        self.case = case
        w, h = case["width"], case["height"]
        g = _gbuffer(1, w, h, seed)
        self.Linear, self.Guide, self.Hit = g["Linear"].view(-1), g["Guide"].view(-1), g["Hit"].view(-1)
        self.mean = g["Mean"].view(-1)
        self.Filtered, self.History, self.Pixels = _f(4 * w * h), self.mean.clone(), _i(w * h)
        C = workloads.base_state(_pick(seed), w, h)
        C[9], C[10] = case["sample"], 1.0 if case["sample"] == 0 else 0.0
        self.C = torch.from_numpy(C).cuda()

    def run(self):
        c = self.case
        self.History.copy_(self.mean)  # the history of the samples before this one
        _check(ab.call("arbor_filterResolve", self.Linear, self.Guide, self.Hit, self.Filtered, self.History, self.Pixels, self.C, c["width"],
                       c["height"]))
        return {"Filtered": self.Filtered, "History": self.History, "Pixels": self.Pixels}


def _weights(seed: int) -> np.ndarray:
    """He-normal weights and small biases, in the library's layout."""
    r = np.random.RandomState(seed % (2 ** 31))
    out = []
    for k, (cin, cout, _) in enumerate(LAYERS):
        out.append((r.standard_normal(cout * 9 * cin) * math.sqrt(2.0 / (9 * cin)) * (0.1 if k == 14 else 1.0)).astype(np.float32))
        out.append((r.standard_normal(cout) * 0.02).astype(np.float32))
    return np.concatenate(out)


class _Net:
    def __init__(self, batch: int, width: int, height: int, seed: int):
        self.lib = ab.lib()
        self.h = ctypes.c_void_p()
        _check(self.lib.arbor_denoiser_create(ctypes.byref(self.h), batch, width, height, 7, ab.stream_handle()))
        p = _weights(seed)
        self.count = p.size
        _check(self.lib.arbor_denoiser_set_params(self.h, p.ctypes.data, p.size))

    def __del__(self):
        try:
            self.lib.arbor_denoiser_destroy(self.h)
        except Exception:
            pass


class _Denoise:
    def __init__(self, case: dict, seed: int):
        self.case = case
        w, h = case["width"], case["height"]
        g = _gbuffer(1, w, h, seed)
        self.g = {k: g[k].view(-1) for k in ("Linear", "Guide", "Normal", "Hit")}
        self.Filtered, self.Denoised = _f(4 * w * h), _f(4 * w * h)
        self.features = torch.zeros(16 * w * h, dtype=torch.int16, device="cuda")
        self.C = torch.from_numpy(workloads.base_state(_pick(seed), w, h)).cuda()
        self.net = _Net(1, w, h, seed)

    def run(self):
        w, h, g = self.case["width"], self.case["height"], self.g
        _check(ab.call("arbor_filterLighting", g["Linear"], g["Guide"], g["Hit"], self.Filtered, self.C, w, h))
        _check(ab.call("arbor_denoiser_features", g["Linear"], g["Guide"], g["Normal"], g["Hit"], self.Filtered, w, h, self.features))
        _check(self.net.lib.arbor_denoiser_infer(self.net.h, self.features.data_ptr(), self.Filtered.data_ptr(), self.Denoised.data_ptr(), w, h))
        return {"Filtered": self.Filtered, "Denoised": self.Denoised}


def _features(g: dict, filtered: torch.Tensor, dtype) -> torch.Tensor:
    """The 16 feature channels of arbor_denoiser_features."""
    l, a, n, h, q = (v.to(dtype) for v in (g["Linear"], g["Guide"], g["Normal"], g["Hit"], filtered))
    depth = torch.log1p(h[..., :1].clamp(0.0, 1.0e4)) * 0.25
    pad = torch.zeros_like(l[..., :3])
    return torch.cat([torch.log1p(l[..., :3].clamp(min=0)), a[..., :3], n[..., :3], depth, torch.log1p(q[..., :3].clamp(min=0)), pad], -1)


class _Train:
    def __init__(self, case: dict, seed: int):
        self.case = case
        n, w, h = case["batch"], case["width"], case["height"]
        g = _gbuffer(n, w, h, seed)
        self.base, self.target = g["Linear"].contiguous(), g["Mean"].contiguous()
        self.features = _features(g, g["Linear"], torch.float32).to(torch.bfloat16).contiguous()
        self.net = _Net(n, w, h, seed)
        self.grad = torch.empty(self.net.count, dtype=torch.float32, pin_memory=True)

    def run(self):
        c = self.case
        loss = ctypes.c_float()
        _check(self.net.lib.arbor_denoiser_gradient(self.net.h, self.features.data_ptr(), self.base.data_ptr(), self.target.data_ptr(), c["batch"],
                                                    c["width"], c["height"], self.grad.data_ptr(), self.grad.numel(), ctypes.byref(loss)))
        return {"gradient": self.grad, "loss": float(loss.value)}


def prepare(case: dict, seed: int):
    kind = case["kind"]
    return {"scene": _Build, "frame": _Frame, "batch": _Batch, "filter": _Filter, "denoise": _Denoise, "train": _Train}[kind](case, seed)


def run(state):
    return state.run()


# -------------------------------------------------------------------- work --
def work(case: dict) -> dict:
    """Bytes: each input read once, each output written once.  Operations of
    the rendering kinds: about 1,500 per primary ray (its cells, the boxes and
    surfaces that hold its nearest hit, one Newton or march solve) and 4,500
    per shadowed pixel (up to four segments, each with the solves of the
    leaves it passes through); of the network: two per multiply-add."""
    kind = case["kind"]
    if kind == "scene":
        n = case["scenes"]
        return {"bytes": 4.0 * n * (2109 * 20 + 32768 * 24 + 2 * 32768 + 65536 * 8 + 64), "flops": n * 32768.0 * 200}
    if kind == "batch":
        sizes = [r for r in workloads.BATCH_RESOLUTIONS if r[0] * r[1] <= case["largest"]]
        px = float(sum(sizes[k % len(sizes)][0] * sizes[k % len(sizes)][1] for k in range(case["views"])))
        return {"bytes": px * 84 + SCENE_BYTES * case["scenes"], "flops": px * (1500 + (4500 if case["shadows"] else 0) + 500)}
    px = float(case["width"] * case["height"])
    if kind == "frame":
        n = case.get("species", 1)
        flops = px * case["spp"] * (1500 + (4500 if case["shadows"] else 0) + 500)
        return {"bytes": SCENE_BYTES * n + px * (16 * 5 + 4) * case["spp"], "flops": flops}
    if kind == "filter":
        return {"bytes": px * (48 + 16 + (16 if case["sample"] else 0) + 16 + 4 + 32), "flops": px * 300}
    if kind == "denoise":
        return {"bytes": px * (64 + 16 + 16), "flops": 2.0 * MACS * px}
    px *= case["batch"]
    return {"bytes": px * (32 + 32) + 4.0 * sum(cin * cout * 9 + cout for cin, cout, _ in LAYERS), "flops": 6.0 * MACS * px}


# ------------------------------------------------------------------- exact --
def _filter64(g: dict, blend: float = 0.86) -> torch.Tensor:
    """filterLighting: the 5x5 same-surface demodulated filter, in 64 bits."""
    lin, gui, hit = g["Linear"].double(), g["Guide"].double(), g["Hit"].double()
    n, h, w, _ = lin.shape
    t, ident, tree = hit[..., 0], hit[..., 1], hit[..., 2]
    tol = torch.clamp(hit[..., 3] * 6.0, min=0.005)
    demod = lin[..., :3] / (gui[..., :3] + 0.02)
    total = torch.zeros_like(demod)
    weight = torch.zeros_like(t)
    for j in range(-2, 3):
        for k in range(-2, 3):
            y0, y1, x0, x1 = max(0, -j), min(h, h - j), max(0, -k), min(w, w - k)
            here = (slice(None), slice(y0, y1), slice(x0, x1))
            there = (slice(None), slice(y0 + j, y1 + j), slice(x0 + k, x1 + k))
            same = (ident[here] == ident[there]) & (tree[here] == tree[there]) & ((t[there] - t[here]).abs() <= tol[here])
            wt = same.double() * math.exp(-0.3 * (j * j + k * k))
            total[here] += demod[there] * wt[..., None]
            weight[here] += wt
    col = lin[..., :3]
    smooth = total / weight.clamp(min=1e-30)[..., None] * (gui[..., :3] + 0.02)
    use = (weight > 0) & (t < FAR)
    col = torch.where(use[..., None], col + (smooth - col) * blend, col)
    return torch.cat([col, torch.ones_like(col[..., :1])], -1)


def _conv64(x: torch.Tensor, wt: torch.Tensor, bias: torch.Tensor, leaky: bool) -> torch.Tensor:
    """3x3 convolution, zero padding, NHWC, as nine products; wt (cout, 9, cin)."""
    n, h, w, _ = x.shape
    p = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1))
    y = bias.expand(n, h, w, -1)
    for tap in range(9):
        y = y + p[:, tap // 3:tap // 3 + h, tap % 3:tap % 3 + w] @ wt[:, tap].T
    return torch.where(y > 0, y, 0.1 * y) if leaky else y


def _network64(x: torch.Tensor, params: list) -> torch.Tensor:
    conv = lambda k, v: _conv64(v, params[2 * k], params[2 * k + 1], bool(LAYERS[k][2]))  # noqa: E731
    pool = lambda v: 0.25 * (v[:, 0::2, 0::2] + v[:, 0::2, 1::2] + v[:, 1::2, 0::2] + v[:, 1::2, 1::2])  # noqa: E731
    up = lambda skip, low: torch.cat([skip, low.repeat_interleave(2, 1).repeat_interleave(2, 2)], -1)  # noqa: E731
    e0 = conv(1, conv(0, x))
    e1 = conv(3, conv(2, pool(e0)))
    e2 = conv(5, conv(4, pool(e1)))
    b3 = conv(7, conv(6, pool(e2)))
    d2 = conv(9, conv(8, up(e2, b3)))
    d1 = conv(11, conv(10, up(e1, d2)))
    d0 = conv(13, conv(12, up(e0, d1)))
    return conv(14, d0)


def _params64(seed: int, dev) -> list:
    flat, out, at = torch.from_numpy(_weights(seed)).double().to(dev), [], 0
    for cin, cout, _ in LAYERS:
        out.append(flat[at:at + cout * 9 * cin].view(cout, 9, cin).clone())
        at += cout * 9 * cin
        out.append(flat[at:at + cout].clone())
        at += cout
    return out


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "filter":
        g = _gbuffer(1, case["width"], case["height"], seed)
        filtered = _filter64(g)
        count = float(case["sample"])
        mean = filtered[..., :3] if count == 0 else g["Mean"][..., :3].double() + (filtered[..., :3] - g["Mean"][..., :3].double()) / (count + 1.0)
        history = torch.cat([mean, torch.full_like(mean[..., :1], count + 1.0)], -1)
        return {"Filtered": filtered.reshape(-1), "History": history.reshape(-1), "Pixels": None}
    if kind == "denoise":
        g = _gbuffer(1, case["width"], case["height"], seed)
        filtered = _filter64(g)
        with torch.no_grad():
            out = _network64(_features(g, filtered, torch.float64), _params64(seed, filtered.device))[..., :3]
        den = torch.expm1(torch.log1p(filtered[..., :3].clamp(min=0)) + out)
        return {"Filtered": filtered.reshape(-1), "Denoised": torch.cat([den, torch.ones_like(den[..., :1])], -1).reshape(-1)}
    if kind == "train":
        g = _gbuffer(case["batch"], case["width"], case["height"], seed)
        params = [p.requires_grad_(True) for p in _params64(seed, g["Linear"].device)]
        x = _features(g, g["Linear"], torch.float32).to(torch.bfloat16).double()
        out = _network64(x, params)[..., :3]
        pred = torch.log1p(g["Linear"][..., :3].double().clamp(min=0)) + out
        loss = (pred - torch.log1p(g["Mean"][..., :3].double().clamp(min=0))).abs().mean()
        loss.backward()
        return {"gradient": torch.cat([p.grad.reshape(-1) for p in params]), "loss": float(loss.detach())}
    return None
