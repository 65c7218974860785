"""What this renderer is measured on: one pass each of the calls that a user's
program makes, over the sizes and options that it makes them with.

A case is a dict.  Its "kind" names the call:

  frame     one image through Renderer.render (call "render": allocates, waits,
            reads the counters back) or Renderer.render_into (call "into": one
            frame of an animation, queued into buffers that the caller keeps)
  gi        one Monte Carlo GI image with depth of field, render_into
  batch     one launch of a prepared batch of jobs of uneven size
  distance  CalculateDistance at a set of points
  gradient  a depth and shade image with refined roots, and the gradient of a
            loss on them with respect to formula and camera

Scenes: bulb, box (with "zoom": the camera 1e-5 in front of the surface, field
of view 0.5 degrees), menger, hybrid (Mandelbulb, then Menger sponge),
primitives (a Mandelbox joined with a plane, a sphere and a box), kleinian
(a formula whose parameters are passed by settings key).
"""
from __future__ import annotations

import ctypes as C
import math
import random

import numpy as np
import torch

from mandelbulber2_b200 import abi, configs
from mandelbulber2_b200.render import STATS_FIELDS, Renderer, alloc_outputs, outputs_struct

ENGINES = {name: number for number, name in abi.ENGINE_NAMES.items()}
FRAME_OUTPUTS = ("depth", "iters", "hit", "normal", "shade", "ao", "rgb", "rgb8")
GI_OUTPUTS = ("depth", "iters", "hit", "rgb", "rgb8")
BATCH_OUTPUTS = ("depth", "iters", "hit", "normal", "rgb8")
DETAIL = 1e-3  # detail size of the distance queries


# ---- the cases ---------------------------------------------------------------------
def listed() -> list[dict]:
    return [
        # a thumbnail or an interactive preview: latency and launches count
        {"name": "preview_bulb_64", "kind": "frame", "call": "render", "scene": "bulb", "engine": "wavefront_fp32",
         "width": 64, "height": 64, "ao_rays": 0},
        # a still of the default formula, Lambert and hard shadow
        {"name": "bulb_512", "kind": "frame", "call": "into", "scene": "bulb", "engine": "wavefront_fp32",
         "width": 512, "height": 512, "ao_rays": 0},
        # the benchmark frame: Mandelbox in full HD with 16 AO rays
        {"name": "box_1080p_ao16", "kind": "frame", "call": "into", "scene": "box", "engine": "wavefront_fp32",
         "width": 1920, "height": 1080, "ao_rays": 16},
        # a deep zoom, where the automatic engine iterates in FP64
        {"name": "box_zoom_1080p_ao16", "kind": "frame", "call": "into", "scene": "box", "zoom": True,
         "engine": "wavefront_auto", "width": 1920, "height": 1080, "ao_rays": 16},
        # what render() does when no engine is named: plain FP64; a ragged size
        {"name": "box_fp64_801x451_ao4", "kind": "frame", "call": "render", "scene": "box", "engine": "plain_fp64",
         "width": 801, "height": 451, "ao_rays": 4},
        # a scene with primitives, which takes the reference-order iteration
        {"name": "primitives_800x600_ao4", "kind": "frame", "call": "into", "scene": "primitives",
         "engine": "wavefront_auto", "width": 800, "height": 600, "ao_rays": 4},
        # a formula by settings key: the plain engines' extended kernels
        {"name": "kleinian_fp64_320x240_ao4", "kind": "frame", "call": "into", "scene": "kleinian",
         "engine": "plain_fp64", "width": 320, "height": 240, "ao_rays": 4},
        # a production still: hybrid fractal, path-traced light, 16 samples a pixel, 4 bounces
        {"name": "hybrid_gi_1080p_16spp", "kind": "gi", "scene": "hybrid", "engine": "wavefront_fp32", "width": 1920,
         "height": 1080, "spp": 16, "bounces": 4},
        # many frames of uneven size at once (thumbnails of a parameter search)
        {"name": "batch_128_jobs", "kind": "batch", "engine": "wavefront_auto", "jobs": 128,
         "jobs_seed": 7},
        # distance queries: a physics or placement step, and a block of a voxel grid
        {"name": "distance_box_4099", "kind": "distance", "scene": "box", "engine": "plain_fp64", "points": 4099},
        {"name": "distance_bulb_1m", "kind": "distance", "scene": "bulb", "engine": "plain_fp64", "points": 1 << 20},
        # one step of an inverse problem: forward image and gradient
        {"name": "gradient_bulb_256", "kind": "gradient", "scene": "bulb", "width": 256, "height": 256},
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng: random.Random) -> dict:
    kind = rng.choice(["frame", "frame", "frame", "frame", "gi", "batch", "distance", "distance", "gradient"])
    if kind == "distance":
        return {"kind": kind, "scene": rng.choice(["bulb", "box", "menger", "hybrid"]),
                "engine": rng.choice(["plain_fp64", "plain_fp64", "plain_fp64_strict", "plain_mixed"]),
                "points": _log_int(rng, 1000, 1 << 21)}
    if kind == "gradient":
        side = _log_int(rng, 64, 512)
        return {"kind": kind, "scene": rng.choice(["bulb", "box"]), "width": side, "height": max(48, side - rng.randrange(9))}
    if kind == "batch":
        return {"kind": kind, "engine": rng.choice(["wavefront_auto", "wavefront_fp32"]), "jobs": _log_int(rng, 8, 160),
                "jobs_seed": rng.randrange(1, 1000)}
    width = _log_int(rng, 64, 1920)
    height = max(36, int(width * rng.choice([9 / 16, 3 / 4, 1.0 if width < 1400 else 9 / 16])) - rng.randrange(3))
    if kind == "gi":
        return {"kind": kind, "scene": "hybrid", "engine": "wavefront_fp32", "width": width, "height": height,
                "spp": rng.choice([1, 2, 4, 7, 16]), "bounces": rng.choice([1, 2, 4])}
    case = {"kind": kind, "call": rng.choice(["render", "into", "into"]),
            "scene": rng.choice(["bulb", "bulb", "box", "box", "box", "menger", "hybrid", "primitives", "kleinian"]),
            "width": width, "height": height, "ao_rays": rng.choice([0, 1, 4, 16])}
    if case["scene"] == "kleinian":
        case["engine"] = rng.choice(["plain_fp64", "plain_mixed"])
        case["width"], case["height"] = max(64, width // 3), max(36, height // 3)
    elif case["scene"] in ("hybrid", "primitives"):
        case["engine"] = rng.choice(["plain_fp64", "wavefront_fp32", "wavefront_auto"])
    else:
        case["engine"] = rng.choice(["plain_fp64", "plain_fp64_strict", "plain_mixed", "wavefront_fp32",
                                     "wavefront_fp32", "wavefront_fp64", "wavefront_auto"])
        if case["scene"] == "box" and case["engine"] in ("wavefront_fp64", "wavefront_auto") and rng.random() < 0.5:
            case["zoom"] = True
    return case


# ---- scenes and cameras ----------------------------------------------------------------
BULB = {"formula": "bulb", "power": 8.0, "maxiter": 250, "bailout": 10.0}
BOX = {"formula": "box", "scale": -1.5, "min_r": 0.5, "maxiter": 50, "bailout": 100.0}
MENGER = {"formula": "menger", "maxiter": 12, "bailout": 10.0}
PARTS = {"bulb": BULB, "box": BOX, "menger": MENGER}
DISTANCE_FROM_CAMERA = {"bulb": 3.0, "box": 6.0, "menger": 3.6, "hybrid": 3.0, "primitives": 6.5}


def _scene(name: str) -> abi.Scene:
    if name == "bulb":
        return configs.mandelbulb_scene(8.0, 250)
    if name == "box":
        return configs.mandelbox_scene(-1.5, 0.5, 50)
    if name == "menger":
        return configs.menger_scene(12)
    if name == "hybrid":
        return configs.hybrid_scene()
    if name == "primitives":
        sc = configs.mandelbox_scene(-1.8, 0.5, 40)
        plane = abi.primitive_defaults(abi.PRIMITIVE_PLANE)
        plane.position[:] = [0.0, 0.0, -2.2]
        ball = abi.primitive_defaults(abi.PRIMITIVE_SPHERE)
        ball.position[:] = [2.1, 0.6, -0.4]
        ball.radius = 0.7
        box = abi.primitive_defaults(abi.PRIMITIVE_BOX)
        box.position[:] = [-2.2, 0.3, -0.8]
        box.size[:] = [0.8, 1.2, 0.6]
        box.rotation[:] = [10.0, 0.0, 35.0]
        box.rounding = 0.05
        sc.n_primitives = 3
        for i, q in enumerate((plane, ball, box)):
            sc.primitive[i] = q
        return sc
    if name == "kleinian":
        sc = abi.scene_defaults(abi.FORMULA_PSEUDO_KLEINIAN)
        sc.formula_maxiter = 60
        sc.fractal[0].set_param("analyticDE_tweak_005", 0.076923)
        sc.fractal[0].set_param("transf_addition_constant_0777", [0.173077, 0.307692, 1.0])
        sc.fractal[0].set_param("transf_minimum_radius_05", 0.230769)
        return sc
    raise ValueError(name)


def _view(case: dict, seed: int):
    """Camera position, target and field of view: the scene seen from an angle taken from the seed."""
    rng = random.Random(seed * 7919 + 1)
    if case["scene"] == "kleinian":  # an interior view, the position moved a little
        off = [rng.uniform(-0.004, 0.004) for _ in range(3)]
        pos = (2.12066528836305, -3.70836995527439, 1.90220668159675)
        aim = (2.12183734234493, -3.70761659259838, 1.90598160360012)
        return tuple(a + o for a, o in zip(pos, off)), tuple(a + o for a, o in zip(aim, off)), 53.0
    turn = rng.uniform(-0.12, 0.12)
    dist = DISTANCE_FROM_CAMERA[case["scene"]]
    up = 1.2 if case["scene"] in ("menger", "primitives") else 0.0
    pos = (dist * math.sin(turn), -dist * math.cos(turn), up)
    if not case.get("zoom"):
        return pos, (0.0, 0.0, 0.0), 53.0
    # 1e-5 in front of the point where the ray to the origin meets the surface
    n = math.sqrt(sum(v * v for v in pos))
    d = [-v / n for v in pos]
    t = 0.0
    for _ in range(2000):
        step = _box_distance_at([p + t * v for p, v in zip(pos, d)])
        if step < 1e-12:
            break
        t += 0.5 * step
    hit = [p + t * v for p, v in zip(pos, d)]
    return tuple(h - 1e-5 * v for h, v in zip(hit, d)), tuple(h + v for h, v in zip(hit, d)), 0.5


def _box_distance_at(p) -> float:
    z, de = list(p), 1.0
    for _ in range(BOX["maxiter"]):
        z = [math.copysign(2.0, v) - v if abs(v) > 1.0 else v for v in z]
        r2 = sum(v * v for v in z)
        f = 1.0 / BOX["min_r"] ** 2 if r2 < BOX["min_r"] ** 2 else (1.0 / r2 if r2 < 1.0 else 1.0)
        z = [v * f * BOX["scale"] + c for v, c in zip(z, p)]
        de = de * f * abs(BOX["scale"]) + 1.0
        if sum(v * v for v in z) > BOX["bailout"] ** 2:
            break
    return math.sqrt(sum(v * v for v in z)) / de


def _camera(case: dict, seed: int) -> abi.Camera:
    pos, aim, fov = _view(case, seed)
    if case["kind"] == "gradient":  # the adjoint takes a camera given by its angles
        cam = configs.camera(pos, fov=fov, width=case["width"], height=case["height"])
        cam.use_angles = 1
        cam.angles[:] = [math.atan2(-pos[1], -pos[0]) - 0.5 * math.pi, 0.0, 0.0]
        return cam
    return configs.camera(pos, target=aim, fov=fov, width=case["width"], height=case["height"])


def _params(case: dict, seed: int) -> abi.RenderParams:
    p = configs.base_params(5, 20.0)
    p.seed = seed & 0xFFFF
    if case["kind"] == "gi":
        _, _, p = configs.hybrid_gi_2160p(case["width"], case["height"], spp=case["spp"])
        p.gi_bounces = case["bounces"]
        p.gi_seed = seed & 0xFFFF
    elif case["kind"] == "gradient":
        _, _, p = configs.adjoint_256(case["scene"] if case["scene"] == "box" else "mandelbulb")
    elif case["ao_rays"]:
        p.ao_rays = case["ao_rays"]
        p.ao_seed = 1234 + (seed & 0xFFFF)
        p.light_intensity = 0.6
        p.ambient_intensity = 0.4
    return p


def _points(case: dict, seed: int) -> torch.Tensor:
    """Points of a cube around the solid, its inside and outside."""
    half = {"bulb": 1.3, "box": 3.0, "menger": 1.3, "hybrid": 1.3}[case["scene"]]
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.rand(case["points"], 3, generator=g, dtype=torch.float64, device="cuda") * 2.0 - 1.0) * half


def _weights(case: dict, seed: int):
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = case["width"] * case["height"]
    return [torch.rand(n, generator=g, dtype=torch.float32, device="cuda") + 0.5 for _ in range(2)]


# ---- the calls --------------------------------------------------------------------------
class _Batch:
    """A prepared batch, given back with the state that holds it."""

    def __init__(self, r: Renderer, case: dict, seed: int):
        # sizes, formulas and radii are the case's; the cameras are turned about the z axis by the seed
        scenes, cams, offsets, total = configs.batch_jobs(case["jobs"], seed=case["jobs_seed"])
        turn = random.Random(seed).uniform(-0.3, 0.3)
        for c in cams:
            x, y, z = c.camera[:]
            c.camera[:] = [x * math.cos(turn) - y * math.sin(turn), x * math.sin(turn) + y * math.cos(turn), z]
        p = configs.base_params(5, 20.0)
        p.seed = seed & 0xFFFF
        jobs = (abi.Job * len(cams))()
        for i, c in enumerate(cams):
            jobs[i].camera = c
            jobs[i].scene_index = i
            jobs[i].pixel_offset = offsets[i]
        self.r, self.lib = r, r.lib
        self.bufs = alloc_outputs(total, r.device, BATCH_OUTPUTS)
        self.stats = torch.zeros(len(STATS_FIELDS), dtype=torch.int64, device=r.device)
        o = outputs_struct(self.bufs, self.stats)
        arr = (abi.Scene * len(scenes))(*scenes)
        self.handle = C.c_void_p()
        r._check(self.lib.mbr_batch_create(r.ctx, arr, len(scenes), jobs, len(cams), C.byref(p), C.byref(o),
                                           ENGINES[case["engine"]], None, C.byref(self.handle)))

    def launch(self) -> None:
        s = torch.cuda.current_stream(self.r.device)
        self.r._check(self.lib.mbr_batch_launch(self.handle, C.c_void_p(s.cuda_stream)))

    def __del__(self):
        if self.handle:
            torch.cuda.synchronize(self.r.device)
            self.lib.mbr_batch_destroy(self.handle)
            self.handle = None


def prepare(case: dict, seed: int) -> dict:
    r = Renderer(0)
    s = {"case": case, "r": r}
    if case["kind"] == "batch":
        s["batch"] = _Batch(r, case, seed)
        return s
    r.set_scene(_scene(case["scene"]))
    if case["kind"] == "distance":
        s["points"] = _points(case, seed)
        return s
    s["camera"], s["params"] = _camera(case, seed), _params(case, seed)
    if case["kind"] == "gradient":
        s["w_depth"], s["w_shade"] = _weights(case, seed)
        s["bufs"] = alloc_outputs(case["width"] * case["height"], r.device, ("depth", "hit", "shade"))
    elif case.get("call") != "render":
        names = GI_OUTPUTS if case["kind"] == "gi" else FRAME_OUTPUTS
        s["bufs"] = alloc_outputs(case["width"] * case["height"], r.device, names)
        s["stats"] = torch.zeros(len(STATS_FIELDS), dtype=torch.int64, device=r.device)
    return s


def run(s: dict):
    case, r = s["case"], s["r"]
    if case["kind"] == "batch":
        s["batch"].launch()
        return s["batch"].bufs
    if case["kind"] == "distance":
        return r.distance(s["points"], DETAIL, False, ENGINES[case["engine"]])
    if case["kind"] == "gradient":
        r.render_into(s["camera"], s["params"], s["bufs"], None, abi.ENGINE_PLAIN_MIXED)
        grad = r.adjoint(s["camera"], s["params"], s["bufs"]["depth"], s["bufs"]["hit"], s["w_depth"], s["w_shade"],
                         abi.ENGINE_PLAIN_FP64)
        return {"depth": s["bufs"]["depth"], "shade": s["bufs"]["shade"], "grad": grad}
    if case.get("call") == "render":
        return r.render(s["camera"], s["params"], ENGINES[case["engine"]], FRAME_OUTPUTS).buffers
    r.render_into(s["camera"], s["params"], s["bufs"], s["stats"], ENGINES[case["engine"]])
    return s["bufs"]


# ---- what a pass cannot do without ---------------------------------------------------------
# Operations of one formula iteration that are not by a structural zero, and
# formula iterations of one unit (a pixel without AO; one AO ray of a pixel; a
# path; a point), counted over the scenes' own views.
ITERATION_FLOPS = {"bulb": 26.5, "box": 25.4, "menger": 12.6, "hybrid": 16.0, "primitives": 25.4, "kleinian": 40.0}
PIXEL_ITERATIONS = {"bulb": 70.0, "box": 270.0, "menger": 150.0, "hybrid": 130.0, "primitives": 260.0,
                    "kleinian": 400.0}
AO_ITERATIONS = {"bulb": 15.0, "box": 60.0, "menger": 40.0, "hybrid": 20.0, "primitives": 50.0, "kleinian": 100.0}
ZOOM_PIXEL_ITERATIONS, ZOOM_AO_ITERATIONS = 800.0, 160.0
PATH_ITERATIONS = {1: 200.0, 2: 260.0, 4: 350.0}
POINT_ITERATIONS = {"bulb": 30.0, "box": 12.0, "menger": 6.0, "hybrid": 6.0}
BATCH_JOB_PIXELS, BATCH_PIXEL_ITERATIONS = 279347.0, 140.0
PIXEL_BYTES = {"frame": 8 + 4 + 1 + 12 + 4 + 4 + 12 + 3, "gi": 8 + 4 + 1 + 12 + 3, "gradient": 8 + 1 + 4 + 2 * 4,
               "batch": 8 + 4 + 1 + 12 + 3}


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "batch":
        n = case["jobs"] * BATCH_JOB_PIXELS
        return {"bytes": n * PIXEL_BYTES[kind], "flops": n * BATCH_PIXEL_ITERATIONS * 26.0}
    if kind == "distance":
        n = case["points"]
        return {"bytes": n * 36.0, "flops": n * POINT_ITERATIONS[case["scene"]] * ITERATION_FLOPS[case["scene"]]}
    n = float(case["width"] * case["height"])
    per = ITERATION_FLOPS[case["scene"]]
    if kind == "gi":
        flops = n * case["spp"] * PATH_ITERATIONS[case["bounces"]] * per
    elif kind == "gradient":  # the image, then seven estimates with six tangents at each hit
        flops = n * per * (PIXEL_ITERATIONS[case["scene"]] + 0.4 * 7 * 7 * 4)
    elif case.get("zoom"):
        flops = n * per * (ZOOM_PIXEL_ITERATIONS + case["ao_rays"] * ZOOM_AO_ITERATIONS)
    else:
        flops = n * per * (PIXEL_ITERATIONS[case["scene"]] + case["ao_rays"] * AO_ITERATIONS[case["scene"]])
    return {"bytes": n * PIXEL_BYTES[kind], "flops": flops}


# ---- the same in 64 bits, in plain torch ---------------------------------------------------
# The Mandelbulb, Mandelbox and Menger sponge, marched, refined, shaded and
# occluded as the engines do it, with every quantity in 64 bits.
def _orbit(f: dict, p: torch.Tensor, power=None):
    """|z|, the derivative and whether the orbit left, at points p (n x 3); differentiable."""
    n = p.shape[0]
    ids = torch.arange(n, device=p.device)
    z, c, de = p, p, torch.ones(n, dtype=torch.float64, device=p.device)
    pw = power if power is not None else torch.full((n,), float(f.get("power", 0.0)), dtype=torch.float64, device=p.device)
    got = []
    for i in range(f["maxiter"]):
        x, y, w = z[:, 0], z[:, 1], z[:, 2]
        if f["formula"] == "bulb":
            r = torch.sqrt(x * x + y * y + w * w)
            th, ph = torch.asin(w / r) * pw, torch.atan2(y, x) * pw
            rp = torch.pow(r, pw - 1.0)
            de = rp * de * pw + 1.0
            rp = rp * r
            z = torch.stack([torch.cos(th) * torch.cos(ph) * rp, torch.cos(th) * torch.sin(ph) * rp, torch.sin(th) * rp], 1) + c
        elif f["formula"] == "box":
            z = torch.where(z.abs() > 1.0, torch.copysign(torch.full_like(z, 2.0), z) - z, z)
            r2 = (z * z).sum(1)
            m2 = f["min_r"] ** 2
            k = torch.where(r2 < m2, torch.full_like(r2, 1.0 / m2), torch.where(r2 < 1.0, 1.0 / r2, torch.ones_like(r2)))
            z = z * k[:, None] * f["scale"] + c
            de = de * k * abs(f["scale"]) + 1.0
        else:
            z = torch.sort(z.abs(), dim=1, descending=True)[0] * 3.0
            z = z - torch.stack([torch.full_like(x, 2.0), torch.full_like(x, 2.0), torch.where(z[:, 2] > 1.0, 2.0, 0.0).to(x)], 1)
            de = de * 3.0
        r = torch.sqrt((z * z).sum(1))
        out = ~(r <= f["bailout"])
        last = i + 1 == f["maxiter"]
        done = torch.ones_like(out) if last else out
        if bool(done.any()):
            got.append((ids[done], r[done], de[done], out[done]))
            keep = ~done
            ids, z, c, de, pw = ids[keep], z[keep], c[keep], de[keep], pw[keep]
        if not ids.numel():
            break
    at = torch.cat([g[0] for g in got])
    back = torch.empty_like(at)
    back[at] = torch.arange(n, device=p.device)
    return [torch.cat([g[k] for g in got])[back] for k in (1, 2, 3)]


def _distance(f: dict, p: torch.Tensor) -> torch.Tensor:
    out = []
    for q in p.split(1 << 22):
        r, de, _ = _orbit(f, q)
        out.append(_estimate(f, r, de).clamp(0.0, 10.0))
    return torch.cat(out) if out else torch.empty(0, dtype=torch.float64, device=p.device)


def _estimate(f: dict, r, de):
    if f["formula"] == "bulb":
        return torch.where(r > 1.0, 0.5 * r * torch.log(r) / de, torch.zeros_like(r))
    return r / de if f["formula"] == "box" else (r - 2.0) / de


def _shr(v: torch.Tensor, n: int) -> torch.Tensor:
    return (v >> n) & ((1 << (64 - n)) - 1)


def _wrap(v: int) -> int:
    v &= (1 << 64) - 1
    return v - (1 << 64) if v >> 63 else v


class _ParkMiller:
    def __init__(self, ray: torch.Tensor, seed: int):
        h = ((ray + 1) * _wrap(0x9E3779B97F4A7C15)) ^ _wrap(seed * 0xC2B2AE3D27D4EB4F)
        h = h ^ _shr(h, 29)
        m = 2147483646
        self.s = (2 * (_shr(h, 1) % m) + (h & 1)) % m + 1
        for _ in range(10):
            self.next()

    def next(self) -> torch.Tensor:
        lo, hi = 16807 * (self.s & 0xFFFF), 16807 * (self.s >> 16)
        lo = lo + ((hi & 0x7FFF) << 16) + (hi >> 15)
        self.s = torch.where(lo > 2147483647, lo - 2147483647, lo)
        return self.s


class _Pcg32:
    def __init__(self, state: int, stream: torch.Tensor):
        self.inc = (stream << 1) | 1
        self.s = self.inc + state
        self.s = self.s * 6364136223846793005 + self.inc

    def uniform(self) -> torch.Tensor:
        old = self.s
        self.s = old * 6364136223846793005 + self.inc
        x = _shr(_shr(old, 18) ^ old, 27) & 0xFFFFFFFF
        rot = _shr(old, 59)
        x = ((x >> rot) | (x << ((32 - rot) & 31))) & 0xFFFFFFFF
        return (x >> 8).double() / 16777216.0


def _rays(case: dict, seed: int):
    """Position and the unit view vectors of every pixel; yaw and the vectors before the rotation."""
    pos, aim, fov = _view(case, seed)
    w, h = case["width"], case["height"]
    fwd = np.array(aim) - np.array(pos)
    fwd /= np.linalg.norm(fwd)
    yaw, pitch = math.atan2(fwd[1], fwd[0]) - 0.5 * math.pi, math.atan2(fwd[2], math.hypot(fwd[0], fwd[1]))
    if case["kind"] == "gradient":
        pitch = 0.0
    f = 2.0 * math.tan(fov / 360.0 * math.pi)
    x = torch.arange(w, dtype=torch.float64, device="cuda")
    y = torch.arange(h, dtype=torch.float64, device="cuda")
    ix = (x / w - 0.5) * (w / h) * f
    iy = (0.5 - y / h) * f
    v = torch.stack([ix[None, :].expand(h, w), torch.ones(h, w, dtype=torch.float64, device="cuda"), iy[:, None].expand(h, w)], 2)
    v = v.reshape(-1, 3)
    v = v / v.norm(dim=1, keepdim=True)
    d = v @ torch.tensor(_turn(yaw, pitch), dtype=torch.float64, device="cuda").T
    return torch.tensor(pos, dtype=torch.float64, device="cuda"), d / d.norm(dim=1, keepdim=True), f, yaw, pitch, v


def _turn(yaw: float, pitch: float) -> np.ndarray:
    cz, sz, cx, sx = math.cos(yaw), math.sin(yaw), math.cos(pitch), math.sin(pitch)
    return np.array([[cz, -sz, 0.0], [sz, cz, 0.0], [0.0, 0.0, 1.0]]) @ np.array([[1.0, 0.0, 0.0], [0.0, cx, -sx], [0.0, sx, cx]])


def _march(f, case, p, cam, d, c0):
    """The primary march: t, threshold and whether there is a hit, for every ray."""
    n = d.shape[0]
    t = torch.zeros(n, dtype=torch.float64, device=d.device)
    thr = torch.zeros_like(t)
    hit = torch.zeros(n, dtype=torch.bool, device=d.device)
    low = torch.zeros_like(t)
    step_of, dist_of = torch.zeros_like(t), torch.zeros_like(t)
    rng = _ParkMiller(torch.arange(n, device=d.device), p.seed) if p.jitter else None
    ids = torch.arange(n, device=d.device)
    for _ in range(p.max_raymarching_steps):
        q = cam + d[ids] * t[ids, None]
        th = (q - cam).norm(dim=1) * c0
        dist = _distance(f, q)
        found = dist < th
        hit[ids[found]] = True
        thr[ids[found]], dist_of[ids[found]] = th[found], dist[found]
        ids, dist, th = ids[~found], dist[~found], th[~found]
        if not ids.numel():
            break
        jit = 1.0
        if rng is not None:
            rng.s = rng.s[~found]
            jit = 1.0 - (rng.next() % 1001).double() / 10000.0
        step = ((dist - 0.5 * th) * p.de_factor * jit).clamp(max=3.0)
        low[ids] = t[ids]
        t[ids] += step
        step_of[ids] = step
        inside = t[ids] <= p.view_distance_max
        ids = ids[inside]
        if rng is not None:
            rng.s = rng.s[inside]
        if not ids.numel():
            break
    ids = hit.nonzero()[:, 0]
    if p.refine == abi.REFINE_ROOT:
        lo, hi = low[ids], t[ids].clone()
        going = hi > lo
        for _ in range(p.binary_steps):
            mid = 0.5 * (lo + hi)
            going = going & (mid > lo) & (mid < hi)
            if not bool(going.any()):
                break
            q = cam + d[ids] * mid[:, None]
            under = _distance(f, q) < (q - cam).norm(dim=1) * c0
            hi = torch.where(going & under, mid, hi)
            lo = torch.where(going & ~under, mid, lo)
        t[ids] = hi
        thr[ids] = hi * c0
    else:
        going, step, window = torch.ones_like(ids, dtype=torch.bool), step_of[ids] * 0.5, 1.0 - 0.001 * p.detail_level
        tt, th, dist = t[ids], thr[ids], dist_of[ids]
        for _ in range(p.binary_steps):
            going = going & ~((dist < th) & (dist > th * window))
            tt = torch.where(going & (dist > th), tt + step, torch.where(going & (dist < th * window), tt - step, tt))
            q = cam + d[ids] * tt[:, None]
            th = torch.where(going, (q - cam).norm(dim=1) * c0, th)
            dist = torch.where(going, _distance(f, q), dist)
            step = step * 0.5
        t[ids], thr[ids] = tt, th
    return t, thr, ids


def _normals(f, q, delta):
    g = []
    for a in range(3):
        e = torch.zeros(3, dtype=torch.float64, device=q.device)
        e[a] = 1.0
        g.append(_distance(f, q + e * delta[:, None]) - _distance(f, q - e * delta[:, None]))
    g = torch.stack(g, 1)
    norm = g.norm(dim=1, keepdim=True)
    one = torch.tensor([1.0, 0.0, 0.0], dtype=torch.float64, device=q.device)
    return torch.where((g.abs() < 1e-50).all(1, keepdim=True), one, g / norm)


def _walk(f, q, v, start, end, thr, factor, most):
    """Marches from q along v; the share of the way to `end` that is left where it meets the surface (0: it does not)."""
    left = torch.zeros_like(thr)
    ids = (start < end).nonzero()[:, 0]
    t = start.clone()
    for _ in range(most):
        if not ids.numel():
            break
        dist = _distance(f, q[ids] + v[ids] * t[ids, None])
        met = dist < thr[ids].float().double()
        left[ids[met]] = ((end - t) / end)[ids[met]]
        ids, dist = ids[~met], dist[~met]
        t[ids] += (dist * factor).clamp(min=1e-15)
        ids = ids[t[ids] < end[ids]]
    return left


def _cosine(n, u1, u2):
    r, phi = u1.sqrt(), 2.0 * math.pi * u2
    lx, ly, lz = r * phi.cos(), r * phi.sin(), (1.0 - u1).clamp(min=0.0).sqrt()
    x, y, z = n[:, 0], n[:, 1], n[:, 2]
    s = torch.where(z >= 0.0, 1.0, -1.0).to(z)
    a = -1.0 / (s + z)
    b = x * y * a
    return torch.stack([(1.0 + s * x * x * a) * lx + b * ly + x * lz, s * b * lx + (s + y * y * a) * ly + y * lz,
                        -s * x * lx - y * ly + z * lz], 1)


def exact(case: dict, seed: int):
    if case["kind"] in ("gi", "batch") or case["scene"] not in PARTS:
        return None
    f = PARTS[case["scene"]]
    if case["kind"] == "distance":
        return _distance(f, _points(case, seed)), None
    p = _params(case, seed)
    cam, d, fov, yaw, pitch, v0 = _rays(case, seed)
    c0 = fov / case["height"] / p.detail_level
    t, thr, ids = _march(f, case, p, cam, d, c0)
    n = d.shape[0]
    zeros = torch.zeros(n, dtype=torch.float64, device=d.device)
    depth = torch.full_like(zeros, 1e20)
    depth[ids] = t[ids]
    q, th = cam + d[ids] * t[ids, None], thr[ids]
    nrm = _normals(f, q, th * p.smoothness)
    light = torch.tensor(list(p.light_direction), dtype=torch.float64, device=d.device)
    light = light / light.norm()
    lam = (nrm @ light).clamp(min=0.0)
    lam = ((1.0 - p.material_shading + lam * p.material_shading) * p.light_intensity).clamp(max=500.0)
    shade = zeros.clone()
    if p.shadow_enable:
        far = torch.full_like(th, p.view_distance_max)
        open_ = _walk(f, q, light.expand(q.shape[0], 3), th, far, th, p.de_factor, p.max_raymarching_steps) == 0.0
        lam = torch.where((lam > 0.001) & open_, lam, torch.zeros_like(lam))
    shade[ids] = lam
    if case["kind"] == "gradient":
        return {"depth": depth, "shade": shade, "grad": _gradient(f, case, seed, p, cam, d, yaw, v0, c0, t, ids, light)}
    ao = torch.ones_like(zeros)
    if p.ao_rays:
        rng = _Pcg32(p.ao_seed, ids)
        total = torch.zeros_like(th)
        end = (q - cam).norm(dim=1) * fov
        for _ in range(p.ao_rays):
            u1 = rng.uniform()
            v = _cosine(nrm, u1, rng.uniform())
            total += 1.0 - _walk(f, q, v, th, end, th, 2.0, p.max_raymarching_steps)
        ao[ids] = total / p.ao_rays
    normal = torch.zeros(n, 3, dtype=torch.float64, device=d.device)
    normal[ids] = nrm
    rgb = zeros.clone()
    rgb[ids] = p.albedo * (shade[ids] + p.ambient_intensity * ao[ids])
    return {"depth": depth, "iters": None, "hit": None, "normal": normal, "shade": shade, "ao": ao,
            "rgb": rgb[:, None].expand(n, 3), "rgb8": None}


def _gradient(f, case, seed, p, cam, d, yaw, v0, c0, t, ids, light):
    """The gradient of sum(w_depth * depth + w_shade * shade) by the implicit function theorem at the roots:
    power, scale, squared minimum radius, camera position, yaw; the last entry is unused."""
    if f["formula"] != "bulb":
        return None
    wd, ws = (w.double()[ids] for w in _weights(case, seed))
    dirs, tt = d[ids], t[ids]
    q = (cam + dirs * tt[:, None]).detach()

    def estimate(pt, power):
        r, de, left = _orbit(f, pt, power)
        e = _estimate(f, r, de).clamp(0.0, 10.0)
        return torch.where(left, e, e.detach())

    power = torch.full_like(tt, f["power"]).requires_grad_(True)
    x = q.clone().requires_grad_(True)
    dist = estimate(x, power)
    g, gp = torch.autograd.grad(dist.sum(), (x, power))
    thr = (q - cam).norm(dim=1) * c0
    use = ((dist.detach() - thr).abs() <= 1e-6 * thr) & torch.isfinite(g).all(1)
    cz, sz = math.cos(yaw), math.sin(yaw)
    dm = torch.tensor([[-sz, -cz, 0.0], [cz, -sz, 0.0], [0.0, 0.0, 0.0]], dtype=torch.float64, device=d.device)
    moves = torch.zeros(len(tt), 7, 3, dtype=torch.float64, device=d.device)
    for k in range(3):
        moves[:, 3 + k, k] = 1.0
    moves[:, 6] = (v0[ids] @ dm.T) * tt[:, None]
    own = torch.zeros(len(tt), 7, dtype=torch.float64, device=d.device)
    own[:, 0] = gp
    dt = -(own + (g[:, None, :] * moves).sum(2)) / ((g * dirs).sum(1) - c0)[:, None]
    x = q.clone().requires_grad_(True)
    delta = (thr * p.smoothness).detach().requires_grad_(True)
    power = torch.full_like(tt, f["power"]).requires_grad_(True)
    grads = []
    for a in range(3):
        e = torch.zeros(3, dtype=torch.float64, device=d.device)
        e[a] = 1.0
        grads.append(estimate(x + e * delta[:, None], power) - estimate(x - e * delta[:, None], power))
    gv = torch.stack(grads, 1)
    s = (gv @ light) / gv.norm(dim=1)
    s = torch.where(s > 0.0, s, s.detach()) * (p.material_shading * p.light_intensity)
    sx, sd, sp = torch.autograd.grad(s.sum(), (x, delta, power))
    ds = (sx[:, None, :] * (moves + dirs[:, None, :] * dt[:, :, None])).sum(2) + sd[:, None] * c0 * p.smoothness * dt
    ds[:, 0] += sp
    each = torch.where(use[:, None], wd[:, None] * dt + ws[:, None] * ds, torch.zeros_like(dt))
    grad = torch.zeros(abi.GRAD_COUNT, dtype=torch.float64, device=d.device)
    grad[:7] = each.sum(0)
    return grad
