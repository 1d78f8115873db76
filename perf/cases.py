"""Performance cases of the field renderer, through its public entry points.

Each case is one thing a user of the library has it do: point lists for glitch
repair, live-view previews, a view at a new centre, stills in the FP64 form
with and without derivative planes, shallow FP64 views, deep fields of the
other formulas, a whole keyframe ladder in one batched call, an 8K field, and
the video frames composed from two keyframes.  Sizes, centres, caps and zooms
are those of the benchmark workloads and tests (``bench.py``,
``tests/golden/cases.py``), plus odd sizes.

``listed()`` names the fixed cases, ``draw(rng)`` gives further ones of the
same ranges, ``prepare`` makes what a program holds before the call, ``run``
is one pass and ``exact`` the same fields in float64 by plain torch.
"""

from __future__ import annotations

import ctypes
import json
import math
import os
import random

import numpy as np
import torch

import __graft_entry__

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
LADDER_STEP = math.log10(8.0)   # keyframe factor of the 1e100 atlas
TILE_FACTOR = 4.0               # keyframe factor of the song atlas
OVERSCAN = 1.2                  # the song's tiles are this much wider than their view

_shared: dict = {}


def _package():
    return __graft_entry__._package()


def _library():
    if "library" not in _shared:
        _shared["library"] = _package().load_library()
    return _shared["library"]


def _stream():
    """One stream for every call of the program, as the library's per-thread
    scratch wants it."""
    if "stream" not in _shared:
        _shared["stream"] = torch.cuda.Stream()
    return _shared["stream"]


def _handle():
    return ctypes.c_void_p(_stream().cuda_stream)


def _check(status: int) -> None:
    if status != 0:
        raise RuntimeError(_package().native.last_error(_library()))


def _centres() -> dict:
    if "centres" not in _shared:
        with open(os.path.join(ROOT, "tests", "golden", "centres.json"), encoding="ascii") as handle:
            _shared["centres"] = json.load(handle)
    return _shared["centres"]


def _centre(formula: str, key: str):
    """(x, y, julia constant) of a bundled centre, decimal strings."""
    c = _centres()[key]
    return c["re"], c["im"], ((c["c_re"], c["c_im"]) if formula == "julia" else ("0", "0"))


CENTRES = {
    "mandelbrot": ("fhd_stack_e50", "field_e100", "field_640x360_e30"),
    "julia": ("julia_fixed_1", "julia_fixed_2"),
    "burning-ship": ("burning_ship_deep",),
    "tricorn": ("tricorn_deep",),
}


def _log_zoom(case: dict, seed: int) -> float:
    """The case's zoom, moved by up to a quarter of a decade: a camera stops
    anywhere between two keyframes, so each seed is another view."""
    return case["log_zoom"] + 0.25 * random.Random(seed * 7919 + 13).random()


# ------------------------------------------------------------------- cases


def listed() -> list[dict]:
    return [
        # Glitch repair: a short list of flagged pixels rendered as points
        # from a keyframe's reference (host arrays in and out).  The smallest
        # call: launch and copy latency.
        dict(name="points_1000_e27", kind="points", count=1000, centre="fhd_stack_e50", log_zoom=27.0, cap=89000),
        # Live view while dragging or zooming: a small odd-sized preview from
        # a prepared reference, field into host memory (backend 4).
        dict(name="preview_321x181_e45", kind="host", width=321, height=181, centre="fhd_stack_e50", log_zoom=45.0,
             cap=137000),
        # The user picks another place: reference orbit, series and BLA
        # tables for the new centre, the first field, and the handle given
        # back.
        dict(name="new_view_640x360_e60", kind="view", width=640, height=360, centre="field_e100", log_zoom=60.0,
             cap=150000),
        # A single field in the FP64 form with counts, coloured with the
        # built-in palette (the plain single-field workload).
        dict(name="plain_640x360_e30", kind="field", form=0, colour=True, width=640, height=360,
             centre="field_640x360_e30", log_zoom=30.0, cap=50000),
        # A still with the distance estimate: all six render planes into host
        # memory, then the KFP pass over them.
        dict(name="still_960x540_e50", kind="still", width=960, height=540, centre="fhd_stack_e50", log_zoom=50.0,
             cap=100000),
        # The whole-set view that every zoom starts from: FP64 direct
        # iteration with a large interior.
        dict(name="direct_1920x1080_e0", kind="direct", formula="mandelbrot", width=1920, height=1080,
             centre="fhd_stack_e50", log_zoom=0.0, cap=4709),
        # A deep field of another formula with its derivative planes.
        dict(name="ship_853x480_e40", kind="deep", fields="burning-ship", width=853, height=480, log_zoom=40.0,
             cap=100000, planes=True),
        # The uneven mixed batch: a field of each formula in one call, chosen
        # form, with derivative planes.
        dict(name="mixed_1280x720_e24", kind="deep", fields="mandelbrot,julia,burning-ship,tricorn", width=1280,
             height=720, log_zoom=24.0, cap=50000, planes=True),
        # The headline: every keyframe of the 1920x1080 atlas to 1e100 in one
        # batched call replayed as a graph.
        dict(name="atlas_112x1080p_e100", kind="atlas", width=1920, height=1080, first=0, count=112,
             centre="fhd_stack_e50", cap=200000),
        # A poster-size field at full depth (the 8K workload).
        dict(name="poster_7680x4320_e100", kind="field", form=1, colour=False, width=7680, height=4320,
             centre="field_e100", log_zoom=100.0, cap=1000000),
        # One 4K video frame of the song: parent and child tiles composed
        # into a surface, the KFP pass, and the NV12 frame for the encoder.
        dict(name="frame_kfp_3840x2160", kind="frame", palette="kfp", pack="nv12", width=3840, height=2160,
             centre="fhd_stack_e50", log_zoom=30.0, position=0.45),
        # One 1080p video frame in the built-in palette, packed as RGBA.
        dict(name="frame_aurora_1920x1080", kind="frame", palette="aurora", pack="rgba", width=1920, height=1080,
             centre="fhd_stack_e50", log_zoom=60.0, position=0.7),
    ]


def _size(rng: random.Random, low: int, high: int):
    width = int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))
    height = max(1, int(round(width / rng.choice((16 / 9, 16 / 9, 4 / 3, 1.0, 21 / 9, 9 / 16)))))
    return width, height


def draw(rng: random.Random) -> dict:
    kind = rng.choice(("points", "host", "view", "field", "still", "direct", "deep", "deep", "atlas", "frame", "frame"))
    centre = rng.choice(CENTRES["mandelbrot"])
    log_zoom = round(rng.uniform(13.0, 99.0), 3)
    cap = int(round(10.0 ** rng.uniform(4.0, 5.3)))
    if kind == "points":
        return dict(kind=kind, count=int(round(10.0 ** rng.uniform(0.5, 5.5))), centre=centre, log_zoom=log_zoom,
                    cap=cap)
    if kind in ("host", "view"):
        width, height = _size(rng, 64, 1920)
        return dict(kind=kind, width=width, height=height, centre=centre, log_zoom=log_zoom, cap=cap)
    if kind == "still":
        width, height = _size(rng, 160, 1600)
        return dict(kind=kind, width=width, height=height, centre=centre, log_zoom=log_zoom, cap=cap)
    if kind == "field":
        form = rng.choice((0, 1))
        width, height = _size(rng, 96, 3840 if form else 1280)
        return dict(kind=kind, form=form, colour=rng.random() < 0.5, width=width, height=height, centre=centre,
                    log_zoom=log_zoom, cap=cap)
    if kind == "direct":
        formula = rng.choice(("mandelbrot", "mandelbrot", "julia", "burning-ship", "tricorn"))
        width, height = _size(rng, 160, 1920)
        return dict(kind=kind, formula=formula, width=width, height=height, centre=rng.choice(CENTRES[formula]),
                    log_zoom=round(rng.uniform(0.0, 10.5), 3), cap=int(round(10.0 ** rng.uniform(3.0, 4.3))))
    if kind == "deep":
        fields = ",".join(rng.choice(tuple(CENTRES)) for _ in range(rng.randint(1, 3)))
        width, height = _size(rng, 96, 600)
        return dict(kind=kind, fields=fields, width=width, height=height, log_zoom=round(rng.uniform(13.0, 90.0), 3),
                    cap=cap, planes=rng.random() < 0.5)
    if kind == "atlas":
        first, (width, height) = rng.randint(0, 80), _size(rng, 320, 1920)
        return dict(kind=kind, width=width, height=height, first=first, count=rng.randint(4, 32),
                    centre="fhd_stack_e50", cap=200000)
    width, height = _size(rng, 320, 3840)
    return dict(kind=kind, palette=rng.choice(("kfp", "kfp", "aurora")), pack=rng.choice(("nv12", "rgba", "rgb0")),
                width=width // 2 * 2, height=height // 2 * 2, centre="fhd_stack_e50",
                log_zoom=round(rng.uniform(15.0, 90.0), 3), position=round(rng.uniform(0.05, 0.95), 3))


# ------------------------------------------------------------- preparation


def _reference(centre: str, log_zoom: float, cap: int) -> int:
    package = _package()
    x, y, _ = _centre("mandelbrot", centre)
    return package.native.create_reference(_library(), x, y, package.atlas.zoom_text(log_zoom), cap,
                                           package.atlas.precision_bits(x, y, log_zoom), 32, reusable=True)


class _References:
    """Handles of one state, given back with it."""

    def __init__(self, handles):
        self.handles = list(handles)

    def __del__(self):
        torch.cuda.synchronize()
        for handle in self.handles:
            _library().fractal_destroy_reference(handle)


def _ladder(case: dict, seed: int):
    """(level, log10 zoom, cap) of the case's keyframes: the factor-8 ladder
    from a seeded origin, caps as the atlas workload has them."""
    jitter = 0.25 * random.Random(seed * 7919 + 13).random()
    levels = []
    for i in range(case["first"], case["first"] + case["count"]):
        cap = min(case["cap"], max(64, int(2000 + 3000 * min(100.0, (i + 1) * LADDER_STEP))))
        levels.append((i, i * LADDER_STEP + jitter, cap))
    return levels


def _direct_view(case: dict, seed: int):
    """Centre (decimal strings, panned by up to 2% of the view), zoom."""
    rng = random.Random(seed * 104729 + 7)
    log_zoom = _log_zoom(case, seed)
    x, y, julia = _centre(case["formula"], case["centre"])
    span = 2.8 / 10.0 ** log_zoom
    base = (-0.6, 0.0) if case["log_zoom"] < 0.5 and case["formula"] != "julia" else (float(x), float(y))
    cx = base[0] + span * rng.uniform(-0.02, 0.02)
    cy = base[1] + span * rng.uniform(-0.02, 0.02)
    return repr(cx), repr(cy), log_zoom, (float(julia[0]), float(julia[1]))


def _points(case: dict, seed: int):
    """Offsets around the reference centre (mantissas and binary exponents),
    log-polar over one view."""
    rng = np.random.default_rng(seed)
    log_zoom = _log_zoom(case, seed)
    radius = (rng.uniform(-1.5, 0.15, case["count"]) - log_zoom) * math.log2(10.0)
    angle = rng.uniform(0.0, 2.0 * math.pi, case["count"])
    exponents = np.ceil(radius).astype(np.int32)
    magnitude = np.exp2(radius - exponents)
    return log_zoom, magnitude * np.cos(angle), magnitude * np.sin(angle), exponents


def prepare(case: dict, seed: int) -> dict:
    package, library = _package(), _library()
    native, atlas = package.native, package.atlas
    kind = case["kind"]
    state = dict(case=case, kind=kind)
    pixels = case.get("width", 0) * case.get("height", 0)
    if kind == "points":
        log_zoom, real, imag, exponents = _points(case, seed)
        handle = _reference(case["centre"], log_zoom, case["cap"])
        state.update(keep=_References([handle]), handle=handle, zoom=atlas.zoom_text(log_zoom), real=real, imag=imag,
                     exponents=exponents)
    elif kind in ("host", "view", "still", "field"):
        log_zoom = _log_zoom(case, seed)
        state.update(zoom=atlas.zoom_text(log_zoom), log_zoom=log_zoom)
        if kind == "view":
            x, y, _ = _centre("mandelbrot", case["centre"])
            state.update(x=x, y=y, bits=atlas.precision_bits(x, y, log_zoom))
        else:
            handle = _reference(case["centre"], log_zoom, case["cap"])
            state.update(keep=_References([handle]), handle=handle)
        state["options"] = native.RenderOptions(backend=0 if kind == "field" else native.BACKEND_CUDA)
        if kind == "still":
            profile = package.kfp.recipe("differences7")
            state.update(kfp=package.kfp.options(profile), lut=package.kfp.palette_lut(profile))
        if kind == "field":
            state.update(field=torch.empty(pixels, dtype=torch.float32, device="cuda"),
                         counts=torch.empty(pixels, dtype=torch.int32, device="cuda"))
            if case["colour"]:
                state["rgb"] = torch.empty(pixels * 3, dtype=torch.uint8, device="cuda")
    elif kind == "direct":
        x, y, log_zoom, julia = _direct_view(case, seed)
        state.update(x=x.encode("ascii"), y=y.encode("ascii"), zoom=atlas.zoom_text(log_zoom), julia=julia,
                     options=native.RenderOptions(), field=torch.empty(pixels, dtype=torch.float32, device="cuda"),
                     counts=torch.empty(pixels, dtype=torch.int32, device="cuda"))
    elif kind == "deep":
        log_zoom = _log_zoom(case, seed)
        specs, buffers = [], []
        for i, formula in enumerate(case["fields"].split(",")):
            keys = CENTRES[formula]
            x, y, julia = _centre(formula, keys[i % len(keys)])
            specs.append(package.fields.FieldSpec(formula, x, y, log_zoom + i, case["width"], case["height"],
                                                  case["cap"], julia))
            planes = [torch.empty(pixels, dtype=torch.float64, device="cuda") for _ in range(2 * case["planes"])]
            buffers.append([torch.empty(pixels, dtype=torch.float32, device="cuda"),
                            torch.empty(pixels, dtype=torch.int32, device="cuda")] + planes)
        fields = package.fields.FieldSet(library, specs)
        targets = [tuple(t.data_ptr() for t in b) + (() if case["planes"] else (None, None)) for b in buffers]
        state.update(fields=fields, keep=_References(fields.handles), buffers=buffers, targets=targets)
    elif kind == "atlas":
        x, y, _ = _centre("mandelbrot", case["centre"])
        stack = atlas.KeyframeStack(library, x, y, _ladder(case, seed), step=LADDER_STEP)
        keyframes = stack.keyframes
        fields = torch.empty((len(keyframes), pixels), dtype=torch.float32, device="cuda")
        counts = torch.empty((len(keyframes), pixels), dtype=torch.int32, device="cuda")
        targets = [(fields[i].data_ptr(), counts[i].data_ptr()) for i in range(len(keyframes))]
        direct = [i for i, k in enumerate(keyframes) if k.reference is None]
        deep = [i for i, k in enumerate(keyframes) if k.reference is not None]
        state.update(stack=stack, keep=_References(stack.handles), fields=fields, counts=counts, targets=targets,
                     order=direct + deep[::-1])
        # Launch shapes are tuned once for a batch of this class, as a
        # program does before its first step.
        tuned = (case["width"], case["height"], len(keyframes), len(direct))
        if tuned not in _shared.setdefault("tuned", set()):
            stack.render_batch_device(targets, case["width"], case["height"], form=1, stream=_stream().cuda_stream,
                                      graph=True, autotune=True, order=state["order"])
            _shared["tuned"].add(tuned)
    else:
        profile = package.kfp.seeded_profile(4242 + seed % 1000, 16)
        lut = torch.from_numpy(package.kfp.palette_lut(profile)).cuda()
        fmt = package.frames.FORMATS[case["pack"]]
        size = library.fractal_gb300_packed_frame_bytes(case["width"], case["height"], fmt)
        rng = random.Random(seed * 31 + 5)
        zoom = OVERSCAN * TILE_FACTOR ** min(0.98, max(0.02, case["position"] + rng.uniform(-0.02, 0.02)))
        cap = int(384 + 500 * (case["log_zoom"] + 1.0))
        tiles = [_tile(case, seed, level, cap) for level in (0, 1)]
        state.update(tiles=tiles, lut=lut, kfp=package.kfp.options(profile), fmt=fmt, zoom=zoom, cap=cap,
                     fraction=min(1.0, zoom / (TILE_FACTOR * OVERSCAN)),
                     controls=[rng.random() for _ in range(4)], interior=(ctypes.c_int * 3)(0, 0, 0),
                     rgb=torch.empty(pixels * 3, dtype=torch.uint8, device="cuda"),
                     packed=torch.empty(int(size), dtype=torch.uint8, device="cuda"))
    torch.cuda.synchronize()
    return state


def _tile(case: dict, seed: int, level: int, cap: int):
    """A keyframe field as the frame pass meets it, made by plain torch (its
    values are the pass's input and must not depend on the renderer)."""
    log_zoom = _log_zoom(case, seed) + level * math.log10(TILE_FACTOR) - math.log10(OVERSCAN)
    value = _field_values("mandelbrot", case["centre"], log_zoom, case["width"], case["height"], cap)
    return value.to(torch.float32)


# --------------------------------------------------------------------- run


def run(state: dict):
    package, library, case = _package(), _library(), state["case"]
    native, kind = package.native, state["kind"]
    if kind == "points":
        field, _ = native.render_points(library, state["handle"], state["zoom"], state["real"], state["imag"],
                                        state["exponents"], case["cap"])
        return {"field": field}
    if kind == "host":
        return {"field": native.render_reference(library, state["handle"], case["width"], case["height"],
                                                 state["zoom"], case["cap"], options=state["options"])}
    if kind == "view":
        handle = native.create_reference(library, state["x"], state["y"], state["zoom"], case["cap"], state["bits"],
                                         32, reusable=True)
        try:
            field = native.render_reference(library, handle, case["width"], case["height"], state["zoom"],
                                            case["cap"], options=state["options"])
        finally:
            library.fractal_destroy_reference(handle)
        return {"field": field}
    if kind == "still":
        field, planes = native.render_reference(library, state["handle"], case["width"], case["height"],
                                                state["zoom"], case["cap"], options=state["options"], planes=True)
        rgb = native.colourise_kfp_planes(library, field, case["width"], case["height"], case["cap"], state["kfp"],
                                          planes, state["lut"])
        return {"field": field, "rgb": rgb, **planes}
    if kind == "field":
        _check(library.fractal_gb300_render_reference_device(
            state["field"].data_ptr(), state["counts"].data_ptr(), case["width"], case["height"], state["zoom"],
            state["handle"], case["cap"], 3, 256, ctypes.byref(state["options"]), case["form"], _handle()))
        out = {"field": state["field"], "counts": state["counts"]}
        if case["colour"]:
            _check(library.fractal_gb300_colourise_device(
                state["field"].data_ptr(), state["rgb"].data_ptr(), case["width"], case["height"], case["cap"], 0.3,
                0.4, 0.7, 0.5, _handle()))
            out["rgb"] = state["rgb"]
        return out
    if kind == "direct":
        _check(library.fractal_gb300_render_direct_device(
            state["field"].data_ptr(), state["counts"].data_ptr(), case["width"], case["height"], state["zoom"],
            state["x"], state["y"], case["cap"], native.FORMULA_IDS[case["formula"]], *state["julia"],
            ctypes.byref(state["options"]), _handle()))
        return {"field": state["field"], "counts": state["counts"]}
    if kind == "deep":
        state["fields"].render_device(state["targets"], form=1, stream=_stream().cuda_stream, graph=True)
        return state["buffers"]
    if kind == "atlas":
        state["stack"].render_batch_device(state["targets"], case["width"], case["height"], form=1,
                                           stream=_stream().cuda_stream, graph=True, order=state["order"])
        return {"fields": state["fields"], "counts": state["counts"]}
    width, height, cap = case["width"], case["height"], state["cap"]
    parent, child = (t.data_ptr() for t in state["tiles"])
    if case["palette"] == "kfp":
        _check(library.fractal_gb300_atlas_colourise_kfp_raw_device(
            parent, width, height, cap, child, width, height, cap, state["rgb"].data_ptr(), width, height,
            state["zoom"], state["fraction"], OVERSCAN, cap, ctypes.byref(state["kfp"]), state["lut"].data_ptr(),
            state["lut"].shape[0], _handle()))
    else:
        _check(library.fractal_gb300_atlas_colourise_device(
            parent, width, height, cap, child, width, height, cap, state["rgb"].data_ptr(), width, height,
            state["zoom"], state["fraction"], cap, *state["controls"], state["interior"], None, _handle()))
    _check(library.fractal_gb300_pack_frame_device(state["rgb"].data_ptr(), width, height, state["fmt"],
                                                   state["packed"].data_ptr(), _handle()))
    return {"rgb": state["rgb"], "packed": state["packed"]}


# -------------------------------------------------------------------- work


def work(case: dict) -> dict:
    """Outputs written and inputs read once; arithmetic: per deep pixel the
    series (32 complex terms, 8 operations each) and the steps that neither
    series nor blocks can skip (about 40 of 22 operations), per pixel of the
    other formulas about 200 such steps, per direct pixel about 100 steps of
    10, per composed and coloured pixel about 100."""
    kind = case["kind"]
    pixels = case.get("width", 0) * case.get("height", 0)
    deep = 8.0 * 32 + 22.0 * 40
    if kind == "points":
        return {"bytes": 24.0 * case["count"], "flops": deep * case["count"]}
    if kind in ("host", "view"):
        return {"bytes": 4.0 * pixels, "flops": deep * pixels}
    if kind == "still":
        return {"bytes": (4.0 + 48.0 + 3.0) * pixels, "flops": 2.0 * deep * pixels}
    if kind == "field":
        return {"bytes": (8.0 + 3.0 * case["colour"]) * pixels, "flops": deep * pixels}
    if kind == "direct":
        return {"bytes": 8.0 * pixels, "flops": 1000.0 * pixels}
    if kind == "deep":
        formulas = case["fields"].split(",")
        flops = sum(deep if f == "mandelbrot" else 22.0 * 200 for f in formulas)
        return {"bytes": (8.0 + 16.0 * case["planes"]) * pixels * len(formulas), "flops": flops * pixels}
    if kind == "atlas":
        return {"bytes": 8.0 * pixels * case["count"], "flops": deep * pixels * case["count"]}
    packed = {"nv12": 1.5, "rgba": 4.0, "rgb0": 4.0}[case["pack"]]
    zoom = OVERSCAN * TILE_FACTOR ** case["position"]
    return {"bytes": (4.0 / zoom ** 2 + 4.0 + 3.0 + packed) * pixels, "flops": 100.0 * pixels}


# ------------------------------------------------- the same fields in float64


def _fixed(text: str, bits: int) -> int:
    """A decimal string as a fixed-point integer with `bits` binary places."""
    text = text.strip()
    sign = -1 if text.startswith("-") else 1
    whole, _, fraction = text.lstrip("+-").partition(".")
    scale = 10 ** len(fraction)
    return sign * ((int((whole or "0") + fraction) << bits) // scale)


def _orbit(formula: str, x: str, y: str, steps: int):
    """The orbit of the parameter (x, y) in fixed point (Mandelbrot or
    tricorn), rounded to float64, up to its escape (inclusive) or `steps`."""
    bits = 64 + int(3.4 * max(len(x), len(y), 40))
    one = 1 << bits
    cr, ci = _fixed(x, bits), _fixed(y, bits)
    zr = zi = 0
    values = []
    for _ in range(steps + 1):
        values.append((zr / one, zi / one))
        if zr * zr + zi * zi > 4 * one * one:
            break
        cross = (zr * zi) >> (bits - 1)
        zr, zi = ((zr * zr - zi * zi) >> bits) + cr, (-cross if formula == "tricorn" else cross) + ci
    return torch.tensor(values, dtype=torch.float64, device="cuda")


def _perturb(formula: str, orbit, dx, dy, cap: int):
    """Smooth values of the pixels at offsets (dx, dy) from the orbit's
    centre: float64 perturbation step by step with rebasing."""
    out = torch.full_like(dx, float(cap))
    at = torch.arange(dx.numel(), device="cuda")
    cr, ci = dx, dy
    dr, di = torch.zeros_like(dx), torch.zeros_like(dx)
    ref = torch.zeros_like(at)
    count, escape = torch.zeros_like(at), torch.zeros_like(dx)
    last = orbit.shape[0] - 1
    n = 0
    limit = min(cap, 60_000)
    while n < limit and at.numel():
        for _ in range(32):
            if n >= cap:
                break
            n += 1
            z = orbit[ref]
            zr, zi = z[:, 0], z[:, 1]
            nr = 2.0 * (zr * dr - zi * di) + (dr - di) * (dr + di) + cr
            ni = 2.0 * (zr * di + dr * (zi + di))
            ni = (-ni if formula == "tricorn" else ni) + ci
            dr, di = nr, ni
            ref = ref + 1
            z = orbit[ref]
            tr, ti = z[:, 0] + dr, z[:, 1] + di
            m2 = tr * tr + ti * ti
            new = (m2 > 4.0) & (count == 0)
            count = torch.where(new, n, count)
            escape = torch.where(new, m2, escape)
            back = (m2 < dr * dr + di * di) | (ref >= last)
            dr, di = torch.where(back, tr, dr), torch.where(back, ti, di)
            ref = torch.where(back, 0, ref)
        done = count > 0
        out[at[done]] = count[done].to(torch.float64) - torch.log2(0.5 * torch.log(escape[done]))
        keep = ~done
        at, cr, ci, dr, di, ref = at[keep], cr[keep], ci[keep], dr[keep], di[keep], ref[keep]
        count, escape = count[keep], escape[keep]
    return out


def _offsets(log_zoom: float, width: int, height: int):
    """Pixel offsets from the view's centre, by rows from the top."""
    span = 2.8 * 10.0 ** -log_zoom
    x = (torch.arange(width, dtype=torch.float64, device="cuda") - (width - 1) / 2.0) / width * (span * width / height)
    y = -(torch.arange(height, dtype=torch.float64, device="cuda") - (height - 1) / 2.0) / height * span
    return x, y


def _field_values(formula: str, centre: str, log_zoom: float, width: int, height: int, cap: int):
    x, y, _ = _centre(formula, centre)
    orbit = _orbit(formula, x, y, min(cap, 8192))
    dx, dy = _offsets(log_zoom, width, height)
    out = torch.empty(height, width, dtype=torch.float64, device="cuda")
    rows = max(1, 8_000_000 // width)
    for top in range(0, height, rows):
        part = dy[top:top + rows]
        out[top:top + rows] = _perturb(formula, orbit, dx.repeat(part.numel()), part.repeat_interleave(width),
                                       cap).view(-1, width)
    return out.view(-1)


def _direct_values(case: dict, seed: int):
    """Direct float64 iteration of the four maps."""
    cx, cy, log_zoom, julia = _direct_view(case, seed)
    formula, cap = case["formula"], case["cap"]
    dx, dy = _offsets(log_zoom, case["width"], case["height"])
    px = (float(cx) + dx).repeat(case["height"])
    py = (float(cy) + dy).repeat_interleave(case["width"])
    out = torch.full_like(px, float(cap))
    at = torch.arange(px.numel(), device="cuda")
    if formula == "julia":
        zr, zi = px, py
        cr, ci = torch.full_like(px, julia[0]), torch.full_like(px, julia[1])
    else:
        zr, zi, cr, ci = torch.zeros_like(px), torch.zeros_like(px), px, py
    if formula == "mandelbrot":
        q = (px - 0.25) ** 2 + py * py
        inside = (q * (q + px - 0.25) <= 0.25 * py * py) | ((px + 1.0) ** 2 + py * py <= 0.0625)
        at, zr, zi, cr, ci = (t[~inside] for t in (at, zr, zi, cr, ci))
    n = 0
    count, escape = torch.zeros_like(at), torch.zeros_like(zr)
    while n < cap and at.numel():
        for _ in range(32):
            if n >= cap:
                break
            n += 1
            if formula == "burning-ship":
                zr, zi = zr.abs(), zi.abs()
            cross = -2.0 * zr * zi if formula == "tricorn" else 2.0 * zr * zi
            zr, zi = zr * zr - zi * zi + cr, cross + ci
            m2 = zr * zr + zi * zi
            new = (m2 > 4.0) & (count == 0)
            count = torch.where(new, n, count)
            escape = torch.where(new, m2, escape)
        done = count > 0
        out[at[done]] = count[done].to(torch.float64) - torch.log2(0.5 * torch.log(escape[done]))
        keep = ~done
        at, zr, zi, cr, ci, count, escape = (t[keep] for t in (at, zr, zi, cr, ci, count, escape))
    return out


def exact(case: dict, seed: int):
    kind = case["kind"]
    if kind == "frame":
        return None  # bytes only
    if kind == "points":
        log_zoom, real, imag, exponents = _points(case, seed)
        x, y, _ = _centre("mandelbrot", case["centre"])
        orbit = _orbit("mandelbrot", x, y, min(case["cap"], 8192))
        dx = torch.from_numpy(np.ldexp(real, exponents)).cuda()
        dy = torch.from_numpy(np.ldexp(imag, exponents)).cuda()
        return {"field": _perturb("mandelbrot", orbit, dx, dy, case["cap"])}
    if kind == "direct":
        return {"field": _direct_values(case, seed), "counts": None}
    if kind == "deep":
        # No value for two of the formulas: a Julia view's long orbits are
        # chaotic and the burning ship amplifies every rounding where an
        # orbit crosses an axis, so two float64 evaluations that round in
        # another order give other counts there.
        out = []
        for i, formula in enumerate(case["fields"].split(",")):
            value = None
            if formula in ("mandelbrot", "tricorn"):
                value = _field_values(formula, CENTRES[formula][i % len(CENTRES[formula])],
                                      _log_zoom(case, seed) + i, case["width"], case["height"], case["cap"])
            out.append([value] + [None] * (1 + 2 * case["planes"]))
        return out if any(values[0] is not None for values in out) else None
    if kind == "atlas":
        fields = [_field_values("mandelbrot", case["centre"], log_zoom, case["width"], case["height"], cap)
                  for _, log_zoom, cap in _ladder(case, seed)]
        return {"fields": torch.stack(fields), "counts": None}
    value = _field_values("mandelbrot", case["centre"], _log_zoom(case, seed), case["width"], case["height"],
                          case["cap"])
    return {"field": value}
