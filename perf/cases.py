"""What a user has this framework do, as measurable cases.

The calls are those of include/r3dgpu.h with device-resident inputs and
outputs, through the package's binding: a rectified pair matched alone
(``r3dgpu_match_stereo_batch`` of one pair, which ``r3dgpu_match_stereo``
forwards to), many uneven pairs in one call, a view's depth map from its
rectified partners (``r3dgpu_compute_depth_map``), and the two stages after it
(``r3dgpu_refine_depth_map``, ``r3dgpu_filter_depth_maps``).

A case is a dict of plain values; ``kind`` selects the call. Images are seeded
synthetic scenes made on the GPU: blurred noise texture over random planes,
8-bit values lifted by 257 as the image reader does, with sensor noise,
textureless patches and occluded runs where the case asks for them.
"""

from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from regard3d_mvs_b200 import _native
from regard3d_mvs_b200.depth_maps import (CConsistencyStats, CDepthMap, ConsistencyOptions, CRefinementImage,
                                          CRefinementStats, RefinementOptions, c_camera, neighbour_lists)
from regard3d_mvs_b200.multi_view import CViewPair, arc_scene, c_grid, pair_geometry
from regard3d_mvs_b200.types import (CPair, CViewU8, CViewU16, MultiStereoOptions, StereoOptions, SubpixelMethod,
                                     camera_struct, pinhole_struct, to_c_options)


# ------------------------------------------------------------------ the cases
def _match(name, w, h, nd, **kw):
    case = {"name": name, "kind": "match", "w": w, "h": h, "nd": nd, "dmin": 0, "wider": 0, "levels": -1, "radius": 3,
            "margin": 4, "lr_full": True, "subpixel": 2, "uniqueness": 0.0, "masked": False, "patches": False}
    case.update(kw)
    return case


def listed():
    return [
        # A preview-sized pair with the default options: launches and host latency.
        _match("preview_320x240_d64", 320, 240, 64),
        # The plain single-level matcher on a VGA pair (the CPU-runnable configuration of the reference).
        _match("vga_640x480_d128_full", 640, 480, 128, levels=0),
        # The cheap left-right check (diagonal of one volume), parabola fit and uniqueness test, one level.
        _match("diagonal_1280x960_d96", 1280, 960, 96, levels=0, lr_full=False, subpixel=1, uniqueness=0.05),
        # An ordinary rectified pair as the multi-view stage makes them: odd sizes, masks, a wider right
        # image, negative disparities, default options (automatic hierarchy).
        _match("rectified_1601x1203_d144", 1601, 1203, 144, dmin=-17, wider=37, masked=True),
        # A full-range pair of the size of a depth-stage view.
        _match("full_2048x1536_d128", 2048, 1536, 128, levels=0),
        # The four-level hierarchy with +-8 ranges, textureless patches and occlusions.
        _match("hierarchy_3072x2048_d256", 3072, 2048, 256, levels=3, radius=0, margin=8, patches=True),
        # The widest photos of the batch configuration, default options.
        _match("photo_6048x4032_d384", 6048, 4032, 384),
        # Pairs of uneven size and label count in one call, half of them hierarchical.
        {"name": "batch_8", "kind": "batch", "pairs": 8, "wmin": 1024, "wmax": 2600},
        # A view's depth map: four partners rectified, matched in one batch with the default options, combined.
        {"name": "view_1600x1200_4", "kind": "view", "w": 1600, "h": 1200, "partners": 4},
        # Refinement of a depth map against four views: float window terms, 7 x 7 samples.
        {"name": "refine_f32_1024x768", "kind": "refine", "w": 1024, "h": 768, "radius": 3, "step": 1, "fp32": True,
         "partners": 4},
        # The same with the default options (double, 9 x 9 window at every second pixel).
        {"name": "refine_f64_800x600", "kind": "refine", "w": 800, "h": 600, "radius": 4, "step": 2, "fp32": False,
         "partners": 4},
        # The consistency filter of a neighbourhood of five depth maps.
        {"name": "filter_5x1536x1152", "kind": "filter", "w": 1536, "h": 1152, "maps": 5},
    ]


def draw(rng):
    """One more case: mostly single pairs, as in use; costs stay below the largest listed pair's."""
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    p = rng.random()
    if p < 0.65:
        levels = rng.choice([-1, -1, -1, 0, 0, 3])
        nd = log_int(24, 384)
        # Full-range cells bounded by those of the listed 2048 x 1536 pair with half as many labels again.
        wmax = 4096 if levels != 0 else min(3000, int(math.sqrt(2048 * 1536 * 192 / nd * 1.4)))
        w = log_int(300, max(301, wmax))
        h = max(200, int(round(w / rng.choice([1.5, 4.0 / 3.0, 1.25]))))
        case = _match("", w, h, nd, levels=levels, dmin=rng.choice([0, 0, -rng.randrange(1, 40)]),
                      wider=rng.choice([0, 0, rng.randrange(1, 60)]), masked=rng.random() < 0.4,
                      patches=rng.random() < 0.4, subpixel=rng.choice([0, 1, 2, 2]))
        if levels == 3:
            case["radius"], case["margin"] = 0, 8
        if rng.random() < 0.25:
            case["lr_full"], case["uniqueness"] = False, rng.choice([0.0, 0.05])
        del case["name"]
        return case
    if p < 0.75:
        return {"kind": "batch", "pairs": rng.randrange(2, 9), "wmin": 640, "wmax": log_int(900, 2600)}
    if p < 0.85:
        w = log_int(480, 1600)
        return {"kind": "view", "w": w, "h": int(w * 0.75) + rng.randrange(0, 8), "partners": rng.randrange(2, 5)}
    if p < 0.95:
        w = log_int(240, 1024)
        fp32 = rng.random() < 0.5
        return {"kind": "refine", "w": w, "h": int(w * 0.75) + rng.randrange(0, 8), "radius": 3 if fp32 else 4,
                "step": 1 if fp32 else 2, "fp32": fp32, "partners": rng.randrange(1, 5)}
    w = log_int(400, 1536)
    return {"kind": "filter", "w": w, "h": int(w * 0.75) + rng.randrange(0, 8), "maps": rng.randrange(3, 6)}


# ------------------------------------------------------------------ inputs
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFF)


def _blur(t, sigma=1.5):
    r = torch.arange(-5, 6, device="cuda", dtype=torch.float32)
    k = torch.exp(-0.5 * (r / sigma) ** 2)
    k = k / k.sum()
    t = t[None, None]
    t = torch.nn.functional.conv2d(torch.nn.functional.pad(t, (5, 5, 0, 0), mode="replicate"), k.view(1, 1, 1, 11))
    t = torch.nn.functional.conv2d(torch.nn.functional.pad(t, (0, 0, 5, 5), mode="replicate"), k.view(1, 1, 11, 1))
    return t[0, 0]


def _pair_images(seed, wl, wr, h, dmin, nd, patches):
    """Left (h x wl) and right (h x wr) u16 images with x_left - x_right = d of random planes in the range."""
    g = _generator(seed)

    def uniform(lo, hi, *shape):
        return lo + (hi - lo) * torch.rand(*shape, generator=g, device="cuda", dtype=torch.float32)

    lo, hi = dmin + min(5, nd // 4), dmin + nd - min(8, nd // 4)
    off = max(0, -dmin) + 8  # texture column of left column 0
    tw = max(wl, wr + max(hi, 0)) + off + nd + 16
    tex = _blur(uniform(0.0, 255.0, h, tw))
    tex = (tex - tex.min()) * (255.0 / (tex.max() - tex.min()))
    rnd = torch.rand(64, 6, generator=g, device="cuda").cpu().numpy()
    if patches:  # constant patches over about 15 % of the area
        for i in range(30):
            x0, y0 = int(rnd[i, 0] * wl * 0.9), int(rnd[i, 1] * h * 0.9)
            tex[y0:y0 + 8 + int(rnd[i, 2] * 0.14 * h), x0:x0 + 8 + int(rnd[i, 3] * 0.14 * wl)] = 20 + 215 * float(rnd[i, 4])
    ys = torch.arange(h, device="cuda", dtype=torch.float32)[:, None]
    xr = torch.arange(wr, device="cuda", dtype=torch.float32)[None, :]
    slope = (hi - lo) / (2.0 * max(wl, h))
    best = torch.full((h, wr), float("inf"), device="cuda")
    disp = torch.zeros((h, wr), device="cuda")
    for i in range(40, 48):  # 8 planes, each pixel takes the nearest seed's
        sx, sy = float(rnd[i, 0]) * wr, float(rnd[i, 1]) * h
        dist = (xr - sx) ** 2 + (ys - sy) ** 2
        d = lo + (hi - lo) * float(rnd[i, 2]) + slope * (2 * float(rnd[i, 3]) - 1) * (xr - sx) \
            + slope * (2 * float(rnd[i, 4]) - 1) * (ys - sy)
        disp = torch.where(dist < best, d, disp)
        best = torch.minimum(dist, best)
    pos = (xr + disp.clamp(lo, hi) + off).clamp(0, tw - 2)
    x0 = pos.floor()
    i0 = x0.long()
    v = torch.gather(tex, 1, i0) * (1 - (pos - x0)) + torch.gather(tex, 1, i0 + 1) * (pos - x0)
    v = v + 2.0 * torch.randn(h, wr, generator=g, device="cuda")
    if patches:  # occlusions: short runs of fresh noise over about 10 % of the right image
        cells = torch.rand(h, (wr + 15) // 16, generator=g, device="cuda").repeat_interleave(16, 1)[:, :wr] < 0.1
        v = torch.where(cells, uniform(0.0, 255.0, h, wr), v)

    def lift(t):
        return (t.round().clamp(0, 255).to(torch.int32) * 257).to(torch.int16).contiguous()  # u16 bits

    return lift(tex[:, off:off + wl]), lift(v)


def _masks(wl, wr, h):
    """Valid regions of rectified images: slanted left and right borders, a few empty rows."""
    def one(w, lean):
        y = torch.arange(h, device="cuda")[:, None]
        x = torch.arange(w, device="cuda")[None, :]
        ok = (x >= lean * y // 40 + w // 50) & (x < w - (h - y) // 30) & (y >= 3)
        return torch.where(ok, 255, 0).to(torch.uint8).contiguous()

    return one(wl, 2), one(wr, 1)


def _fill_pair(pair, keep, case, seed):
    wl, h, nd, dmin = case["w"], case["h"], case["nd"], case["dmin"]
    wr = wl + case["wider"]
    left, right = _pair_images(seed, wl, wr, h, dmin, nd, case["patches"])
    pair.left = CViewU16(left.data_ptr(), wl, h, wl)
    pair.right = CViewU16(right.data_ptr(), wr, h, wr)
    keep += [left, right]
    if case["masked"]:
        lm, rm = _masks(wl, wr, h)
        pair.left_valid, pair.right_valid = CViewU8(lm.data_ptr(), wl, h, wl), CViewU8(rm.data_ptr(), wr, h, wr)
        keep += [lm, rm]
    pair.disparity_min, pair.num_disparities = dmin, nd
    pair.options = to_c_options(StereoOptions(
        levels=case["levels"], range_radius=case["radius"], range_margin=case["margin"], lr_full_match=case["lr_full"],
        subpixel=SubpixelMethod(case["subpixel"]), uniqueness=case["uniqueness"]))
    disp = torch.empty(h, wl, dtype=torch.float32, device="cuda")
    conf = torch.empty_like(disp)
    pair.out.disparity, pair.out.confidence, pair.out.stride = disp.data_ptr(), conf.data_ptr(), wl
    return disp, conf


def _batch_specs(case, seed):
    """The batch's pairs: widths log-uniform, 3:2 or 4:3, 64 to 384 labels, half with four levels. Sizes do not
    depend on the seed, so that passes on other inputs of the case do the same work."""
    rng = np.random.default_rng(case["pairs"] * 1000 + case["wmax"])
    out = []
    for i in range(case["pairs"]):
        w = int(round(math.exp(rng.uniform(math.log(case["wmin"]), math.log(case["wmax"])))))
        h = int(round(w / (1.5 if rng.random() < 0.5 else 4.0 / 3.0)))
        nd = int((64, 128, 192, 256, 384)[rng.integers(0, 5)])
        kw = {"levels": 3, "radius": 0, "margin": 8} if i % 2 else {"levels": 0}
        out.append(_match("", w, h, nd, **kw))
    return out


def _scene(case, seed, views):
    return arc_scene(n_views=views, width=case["w"], height=case["h"], planes=10, partners=views - 1, seed=seed,
                     arc_deg=100.0 / 31.0 * (views - 1), device="cuda")


def _prepare_view(case, seed, state):
    n = case["partners"] + 1
    scene = _scene(case, seed, n)
    v = scene["views"][n // 2]
    cam = v["camera"]
    w, h = case["w"], case["h"]
    keep = state["keep"]

    def dev(a):
        t = torch.from_numpy(np.ascontiguousarray(a).view(np.int16)).cuda()
        keep.append(t)
        return CViewU16(t.data_ptr(), a.shape[1], a.shape[0], a.shape[1])

    pin = {"model": 0, "width": w, "height": h, "fx": cam["K"][0, 0], "fy": cam["K"][1, 1], "cx": cam["K"][0, 2],
           "cy": cam["K"][1, 2]}
    pairs = (CViewPair * len(v["pairs"]))()
    for q, p in zip(pairs, v["pairs"]):
        q.partner, q.partner_camera = dev(p["image"]), camera_struct(pin)
        q.base_from_rect[:] = [float(x) for x in (cam["R"] @ p["R_rect"].T).ravel()]
        q.partner_from_rect[:] = [float(x) for x in (p["R_partner"] @ p["R_rect"].T).ravel()]
        q.left, q.right = pinhole_struct(p["left"]), pinhole_struct(p["right"])
        # A fixed search range, as a user takes from the scene's depth bounds.
        q.disparity_min, q.num_disparities = p["disparity_min"], p["num_disparities"]
        q.geometry = pair_geometry(cam, p)
    depth = torch.empty(h, w, dtype=torch.float32, device="cuda")
    conf = torch.empty_like(depth)
    mask = torch.empty(h, w, dtype=torch.int16, device="cuda")
    state.update(base=dev(v["image"]), camera=camera_struct(pin), grid=c_grid(cam), pairs=pairs,
                 stereo=to_c_options(StereoOptions()), multi=MultiStereoOptions().c(), cells=ctypes.c_uint64(0),
                 out={"depth": depth, "confidence": conf, "mask": mask}, stride=w)


def _depth_views(case, seed, n):
    """Views of a scene with the depth maps a matcher leaves: the true depth in 4 x 4 blocks with a smooth error of
    up to 1 %, and a few holes and wrong depths; grey images as floats. Returns the views and their cameras."""
    scene = _scene(case, seed, n)
    g = _generator(seed + 77)
    w, h = case["w"], case["h"]
    y = torch.arange(h, device="cuda")[:, None]
    x = torch.arange(w, device="cuda")[None, :]
    out = []
    for v in scene["views"]:
        t = torch.from_numpy(v["depth"]).cuda()
        d = t[(y // 4 * 4 + 2).clamp(max=h - 1), (x // 4 * 4 + 2).clamp(max=w - 1)]
        d = d * (1.0 + 0.004 * torch.sin(x / 9.0) * torch.cos(y / 13.0))
        r = torch.rand(h, w, generator=g, device="cuda")
        d = torch.where(r < 0.02, d * 1.2, d)
        d = torch.where(r > 0.95, torch.zeros_like(d), d)
        K, R, C = v["camera"]["K"], v["camera"]["R"], v["camera"]["C"]
        cam = {"width": w, "height": h, "fx": K[0, 0], "fy": K[1, 1], "cx": K[0, 2], "cy": K[1, 2], "rotation": R,
               "center": C}
        out.append({"camera": cam, "depth": d.float().contiguous(), "image8": torch.from_numpy(v["image8"]).cuda()})
    return out


def _refinement_images(lib, views, w, h, keep):
    imgs = []
    for v in views:
        gray = v["image8"].float().contiguous()
        data = torch.empty(h, w, 3, dtype=torch.float32, device="cuda")
        _native.check(lib, lib.r3dgpu_make_refinement_image(gray.data_ptr(), w, w, h, 0.0, data.data_ptr(), 3 * w, None))
        keep.append(data)
        imgs.append((v["camera"], data))
    return imgs


def _refinement_options(case):
    return RefinementOptions(radius=case["radius"], step=case["step"], fp32=case["fp32"])


def _prepare_refine(case, seed, state):
    w, h = case["w"], case["h"]
    views = _depth_views(case, seed, case["partners"] + 1)
    base = len(views) // 2
    imgs = _refinement_images(state["lib"], views, w, h, state["keep"])

    def c_image(camera, data):
        c = CRefinementImage()
        c.camera, c.data, c.stride = c_camera(camera), data.data_ptr(), 3 * w
        return c

    others = [i for i in range(len(views)) if i != base]
    state.update(input=views[base]["depth"], imgs=imgs, base=base, camera=c_camera(views[base]["camera"]),
                 c_base=c_image(*imgs[base]), c_views=(CRefinementImage * len(others))(*[c_image(*imgs[i]) for i in others]),
                 options=_refinement_options(case).c(), stats=CRefinementStats(), w=w, h=h,
                 out={"depth": torch.empty_like(views[base]["depth"]), "confidence": torch.zeros(h, w, device="cuda")})


def _prepare_filter(case, seed, state):
    w, h, n = case["w"], case["h"], case["maps"]
    views = _depth_views(case, seed, n)
    maps = (CDepthMap * n)()
    depth, support = [], []
    for i, (m, v) in enumerate(zip(maps, views)):
        m.camera = c_camera(v["camera"])
        d, conf = torch.empty_like(v["depth"]), torch.full((h, w), 0.8, device="cuda")
        mask = torch.ones(h, w, dtype=torch.int16, device="cuda")
        sup = torch.zeros(h, w, dtype=torch.uint8, device="cuda")
        color = v["image8"][..., None].expand(h, w, 3).contiguous()
        m.depth, m.confidence, m.pair_mask, m.support, m.color = (t.data_ptr() for t in (d, conf, mask, sup, color))
        m.stride, m.color_stride, m.width, m.height, m.view = w, 3 * w, w, h, i
        others = [j for j in range(n) if j != i]
        m.num_partners = len(others)
        for k, j in enumerate(others):
            m.partners[k] = j
        depth.append(d)
        support.append(sup)
        state["keep"] += [conf, mask, color]
    off, idx = neighbour_lists([[j for j in range(n) if j != i] for i in range(n)])
    state.update(input=[v["depth"] for v in views], maps=maps, n=n, off=off, idx=idx, options=ConsistencyOptions().c(),
                 stats=CConsistencyStats(), out={"depth": depth, "support": support})


def prepare(case, seed):
    lib = _native.load()
    _native.check(lib, lib.r3dgpu_set_device(torch.cuda.current_device()))
    state = {"kind": case["kind"], "lib": lib, "keep": []}
    if case["kind"] in ("match", "batch"):
        specs = [case] if case["kind"] == "match" else _batch_specs(case, seed)
        pairs = (CPair * len(specs))()
        outs = [_fill_pair(q, state["keep"], c, seed * 64 + i) for i, (q, c) in enumerate(zip(pairs, specs))]
        state.update(pairs=pairs, n=len(specs), disparity=[d for d, _ in outs], confidence=[c for _, c in outs])
    elif case["kind"] == "view":
        _prepare_view(case, seed, state)
    elif case["kind"] == "refine":
        _prepare_refine(case, seed, state)
    else:
        _prepare_filter(case, seed, state)
    torch.cuda.synchronize()
    return state


def run(state):
    lib = state["lib"]
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    if state["kind"] in ("match", "batch"):
        _native.check(lib, lib.r3dgpu_match_stereo_batch(state["pairs"], state["n"], stream))
        return {"disparity": state["disparity"], "confidence": state["confidence"],
                "cells": [int(p.out.cells) for p in state["pairs"]]}
    out = state["out"]
    if state["kind"] == "view":
        _native.check(lib, lib.r3dgpu_compute_depth_map(
            ctypes.byref(state["base"]), ctypes.byref(state["camera"]), ctypes.byref(state["grid"]), state["pairs"],
            len(state["pairs"]), ctypes.byref(state["stereo"]), ctypes.byref(state["multi"]), out["depth"].data_ptr(),
            out["confidence"].data_ptr(), out["mask"].data_ptr(), state["stride"], ctypes.byref(state["cells"]), stream))
        return {**out, "cells": int(state["cells"].value)}
    if state["kind"] == "refine":
        # The call refines in place: the unrefined map stays for the next pass.
        out["depth"].copy_(state["input"])
        out["confidence"].zero_()
        _native.check(lib, lib.r3dgpu_refine_depth_map(
            out["depth"].data_ptr(), out["confidence"].data_ptr(), state["w"], ctypes.byref(state["camera"]),
            state["w"], state["h"], ctypes.byref(state["c_base"]), state["c_views"], len(state["c_views"]),
            ctypes.byref(state["options"]), ctypes.byref(state["stats"]), stream))
        return out
    for d, s in zip(out["depth"], state["input"]):
        d.copy_(s)
    _native.check(lib, lib.r3dgpu_filter_depth_maps(
        state["maps"], state["n"], state["off"].ctypes.data, state["idx"].ctypes.data, ctypes.byref(state["options"]),
        ctypes.byref(state["stats"]), stream))
    return {**out, "kept": int(state["stats"].output)}


# ------------------------------------------------------------------ work
# Integer operations of one aggregated cell: Census cost, eight path updates, sum and winner-takes-all.
_OPS_PER_CELL = 66


def _match_work(c):
    wl, wr, h = c["w"], c["w"] + c["wider"], c["h"]
    nd = (c["nd"] + 15) // 16 * 16
    levels = c["levels"]
    if levels < 0:
        levels, w, hh, n = 0, wl, h, c["nd"]
        while levels < 8 and min((w + 1) // 2, (hh + 1) // 2) >= 96 and n > 48:
            w, hh, n, levels = (w + 1) // 2, (hh + 1) // 2, (n + 1) // 2, levels + 1
    width = wl + (wr if c["lr_full"] else 0)
    # Full range at the coarsest level; about one and a half 16-label units per pixel at the finer ones.
    cells = width * h * nd / 8.0 ** levels + sum(width * h * 24 / 4.0 ** i for i in range(levels))
    return {"bytes": 2.0 * (wl + wr) * h + (wl + wr) * h * c["masked"] + 8.0 * wl * h, "flops": _OPS_PER_CELL * cells}


def work(case):
    kind = case["kind"]
    if kind == "match":
        return _match_work(case)
    if kind == "batch":
        parts = [_match_work(c) for c in _batch_specs(case, 0)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    px = float(case["w"] * case["h"])
    if kind == "view":
        n = case["partners"]
        m = _match_work(_match("", case["w"], case["h"], 256, masked=True))
        return {"bytes": px * (2 * (n + 1) + 10), "flops": n * m["flops"]}
    if kind == "refine":
        # The maps (4 B read, 8 B written) and each refinement image once; about 60 operations per window sample
        # and view, in about six evaluations.
        samples = (2 * case["radius"] // case["step"] + 1) ** 2
        return {"bytes": px * (12 + 12 * (case["partners"] + 1)), "flops": px * samples * case["partners"] * 60 * 6}
    # Depth in and out, confidence, mask, support and colour of every map; a projection per pixel and neighbour.
    return {"bytes": px * case["maps"] * (4 + 4 + 4 + 2 + 1 + 3), "flops": px * case["maps"] * (case["maps"] - 1) * 60}


# ------------------------------------------------------------------ 64-bit results
def _centre_warp(view, base):
    """m = K_j R_j R_0^T K_0^-1 and b = K_j R_j (C_0 - C_j) of the plane-induced warp, float64."""
    def K(c):
        return np.array([[c["fx"], 0, c["cx"]], [0, c["fy"], c["cy"]], [0, 0, 1.0]])

    kr = K(view) @ np.asarray(view["rotation"])
    m = kr @ np.asarray(base["rotation"]).T @ np.linalg.inv(K(base))
    b = kr @ (np.asarray(base["center"]) - np.asarray(view["center"]))
    return torch.from_numpy(m).cuda(), torch.from_numpy(b).cuda()


def _exact_refine(case, seed):
    """Gauss-Newton plane refinement in float64: the per-pixel steps of the call, all pixels at once."""
    s = prepare(case, seed)
    o = _refinement_options(case)
    w, h, r = case["w"], case["h"], o.radius
    depth_in = s["input"].double()
    base_cam, base_img = s["imgs"][s["base"]]
    gray = base_img[..., 0].double()
    others = [s["imgs"][i] for i in range(len(s["imgs"])) if i != s["base"]]
    warps = [_centre_warp(c, base_cam) for c, _ in others]
    tables = [d.double() for _, d in others]
    offs = torch.arange(-r, r + 1, o.step, device="cuda")
    oy, ox = [t.reshape(-1) for t in torch.meshgrid(offs, offs, indexing="ij")]
    n = oy.numel()
    depth, conf = depth_in.clone(), torch.zeros_like(depth_in)
    valid = depth_in > 0
    inner = torch.zeros_like(valid)
    inner[r:h - r, r:w - r] = True

    def slope(ax, ay):
        def neighbour(k):
            z = torch.roll(depth_in, shifts=(-k * ay, -k * ax), dims=(0, 1))
            near = (z - depth_in).float().abs().double() <= 0.05 * torch.minimum(z, depth_in)
            return (z > 0) & near, 1.0 / z
        (pl, wp), (mi, wm), w0 = neighbour(1), neighbour(-1), 1.0 / depth_in
        zero = torch.zeros_like(w0)
        return torch.where(pl & mi, 0.5 * (wp - wm), torch.where(pl, wp - w0, torch.where(mi, w0 - wm, zero)))

    slopes = torch.stack([r * slope(1, 0), r * slope(0, 1)], -1)
    todo = (valid & inner).nonzero()
    for part in todo.split(60000):
        y, x = part[:, 0], part[:, 1]
        win = gray[y[:, None] + oy, x[:, None] + ox]
        win = win - win.mean(1, keepdim=True)
        norm2 = (win * win).sum(1)
        keep = norm2 >= o.min_texture ** 2 * n
        y, x, win, norm2 = y[keep], x[keep], win[keep], norm2[keep]
        if not y.numel():
            continue
        n0 = win / norm2.sqrt()[:, None]
        w0 = 1.0 / depth_in[y, x]
        theta0 = torch.cat([w0[:, None], slopes[y, x]], 1)
        one = torch.ones(n, dtype=torch.float64, device="cuda")
        basis = torch.stack([one, ox / r, oy / r], -1)
        qx, qy = (x[:, None] + ox).double(), (y[:, None] + oy).double()

        def evaluate(j, theta):
            m, b = warps[j]
            wq = theta @ basis.T
            hx, hy, hz = (m[i, 0] * qx + m[i, 1] * qy + m[i, 2] + b[i] * wq for i in range(3))
            px, py = hx / hz, hy / hz
            ok = (hz > 0) & (px >= 0) & (py >= 0) & (px < w - 1) & (py < h - 1)
            px, py = torch.where(ok, px, 0.0), torch.where(ok, py, 0.0)
            ix, iy = px.floor().long(), py.floor().long()
            fx, fy = (px - ix)[..., None], (py - iy)[..., None]
            t = tables[j]
            v = (1 - fy) * ((1 - fx) * t[iy, ix] + fx * t[iy, ix + 1]) + fy * ((1 - fx) * t[iy + 1, ix] + fx * t[iy + 1, ix + 1])
            raw = v[..., 0] - v[..., :1].mean(1)
            n2 = (raw * raw).sum(1)
            good = ok.all(1) & (n2 > 1e-6 * n)
            inv = torch.where(good, n2, 1.0).rsqrt()[:, None]
            nq = raw * inv
            ncc = (nq * n0).sum(1)
            dv = (v[..., 1] * (b[0] - px * b[2]) + v[..., 2] * (b[1] - py * b[2])) / torch.where(ok, hz, 1.0)
            a = dv[..., None] * basis
            d = a - a.mean(1, keepdim=True)
            jac = (d - nq[..., None] * (nq[..., None] * d).sum(1, keepdim=True)) * inv[..., None]
            return good, ncc, jac.transpose(1, 2) @ jac, (jac * (nq - n0)[..., None]).sum(1)

        first = [evaluate(j, theta0)[:2] for j in range(len(others))]
        use = torch.stack([g & (c >= o.min_ncc) for g, c in first], 1)
        count = use.sum(1)
        s0 = (torch.stack([c for _, c in first], 1) * use).sum(1) / count.clamp(min=1)
        none = count == 0
        if o.drop_unconfirmed:
            depth[y[none], x[none]] = 0.0
        conf[y[~none], x[~none]] = s0[~none]
        motion = torch.zeros_like(w0)
        for j, (m, b) in enumerate(warps):
            hx, hy, hz = (m[i, 0] * x + m[i, 1] * y + m[i, 2] + b[i] * w0 for i in range(3))
            mo = torch.hypot(b[0] - hx / hz * b[2], b[1] - hy / hz * b[2]) / hz
            motion = torch.maximum(motion, torch.where(use[:, j] & (hz > 0), mo, 0.0))

        def total(theta):
            score, H, g = torch.zeros_like(w0), torch.zeros(len(w0), 3, 3, dtype=w0.dtype, device="cuda"), torch.zeros_like(theta)
            good = ~none
            for j in range(len(others)):
                ok, ncc, Hj, gj = evaluate(j, theta)
                u = use[:, j]
                good = good & (ok | ~u)
                score, H, g = score + ncc * u, H + Hj * u[:, None, None], g + gj * u[:, None]
            return torch.where(good, score / count.clamp(min=1), -math.inf), H, g

        best = theta0
        score, H, g = total(best)
        live = torch.isfinite(score)
        done = ~live
        scale = torch.ones_like(w0)
        eye = torch.eye(3, dtype=torch.float64, device="cuda")
        for _ in range(o.iterations):
            A = H * (1 + 1e-6 * eye) + 1e-12 * eye
            A = torch.where(done[:, None, None], eye, A)
            delta = -torch.linalg.solve_ex(A, g[..., None])[0][..., 0]
            done = done | ~torch.isfinite(delta).all(1)
            mo = motion * delta.abs().sum(1)
            delta = delta / mo.clamp(min=1.0)[:, None] * scale[:, None]
            done = done | (motion * delta.abs().sum(1) < 1e-3)
            cand = torch.where(done[:, None], best, best + delta)
            sc, H2, g2 = total(cand)
            up = (sc > score) & ~done
            best = torch.where(up[:, None], cand, best)
            H, g = torch.where(up[:, None, None], H2, H), torch.where(up[:, None], g2, g)
            score = torch.where(up, sc, score)
            scale = torch.where(up, 1.0, scale * 0.25)
        take = live & (score > s0 + o.min_gain) & (best[:, 0] > 0) & (motion * (best[:, 0] - w0).abs() <= o.max_shift_px)
        depth[y[take], x[take]] = 1.0 / best[take, 0]
        conf[y[take], x[take]] = score[take]
    return {"depth": depth, "confidence": conf}


def exact(case, seed):
    """The 64-bit values of a refined map. The other calls' floats follow from whole numbers (path sums, labels,
    supports) through per-pixel choices between them, so they have no 64-bit value apart from the result itself."""
    return _exact_refine(case, seed) if case["kind"] == "refine" else None
