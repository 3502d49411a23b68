"""The workloads whose speed is kept under measurement.

Each case is a call a user of the package makes, on inputs resident in GPU
memory where the call takes them there: the quality controller's probe
(single and batched), the encoder's transform, the plan renderer,
SSIMULACRA2 against a kept reference and on a pair, the cover search, and
the batched decode of committed streams.  Sizes run from thumbnails to
12-megapixel photographs, odd ones among them.

    listed()             the cases
    draw(rng)            one more of the same ranges
    prepare(case, seed)  inputs and handles, made from the seed
    run(state)           one pass, returning its outputs
    work(case)           bytes and operations the pass cannot do without
    exact(case, seed)    run's outputs in 64-bit arithmetic (plain torch)
"""
from __future__ import annotations

import ctypes as C
import math
from pathlib import Path

import numpy as np
import torch

import jpxl_gb300 as jg
from jpxl_gb300._lib import PlanStruct

STREAMS = Path(__file__).resolve().parent.parent / "tests" / "golden" / "codestream"
# Lossy VarDCT streams of cjxl: grey 128x128 ones (filtered and not, one and
# several passes, an LF frame), of which the seed picks, and RGB ones of other
# sizes (every transform up to 64x64 among them) at fixed places.
GREY_STREAMS = (
    "50_vardct_mixed_gray_128x128_nofilters_d1", "51_vardct_mixed_gray_128x128_nofilters_d4",
    "52_vardct_mixed_gray_128x128_filters_d1", "53_vardct_mixed_gray_128x128_filters_d4",
    "70_progressive_ac_gray_128x128_nofilters", "71_qprogressive_ac_gray_128x128_nofilters",
    "72_lfframe_gray_128x128_nofilters", "73_progressive_all_gray_128x128_nofilters")
RGB_STREAMS = {1: "06_gradient_300x200_lossy", 4: "63_vardct_outofgamut_rgb_64x64_nofilters_d4",
               7: "64_vardct_lfgroupseam_rgb_128x2176_nofilters_d6"}
STREAM_SLOTS = 9  # places 1, 4 and 7 of every nine are the RGB streams
STREAM_PIXELS = (6 * 128 * 128 + 300 * 200 + 64 * 64 + 128 * 2176) / STREAM_SLOTS


def listed() -> list:
    probe = dict(kind="probe", gaborish=True, epf=3, scale=40000)
    return [
        # a thumbnail's quality probe: launches and latency
        dict(probe, name="probe_64x64_rgb8", width=64, height=64, bits=8, precision="fp32"),
        # a web image of odd size
        dict(probe, name="probe_501x333_rgb8", width=501, height=333, bits=8, precision="fp32"),
        # the benchmark's probe, in its headline precision
        dict(probe, name="probe_2048x2048_rgb16", width=2048, height=2048, bits=16,
             precision="bf16x6"),
        # the controller's sweep: uneven frames x eight quantizers in one graph
        dict(name="sweep_8x8_rgb8", kind="sweep", frames=8, width=1600, height=1200, bits=8,
             precision="fp32", lanes=8),
        # encoding a video-sized frame, and a 12 MPix photograph
        dict(name="encode_1920x1080_rgb8", kind="encode", width=1920, height=1080, bits=8,
             precision="fp32", gaborish=True, scale=32768),
        dict(name="encode_4096x3072_rgb16", kind="encode", width=4096, height=3072, bits=16,
             precision="bf16x6", gaborish=True, scale=52000),
        # the renderer's two outputs: 8-bit pixels to show, linear planes to measure
        dict(name="render_1920x1080_srgb8", kind="render", width=1920, height=1080, bits=8,
             precision="fp32", gaborish=True, epf=3, scale=32768, out="srgb8"),
        dict(name="render_777x613_linear", kind="render", width=777, height=613, bits=8,
             precision="bf16x6", gaborish=True, epf=1, scale=30000, out="linear"),
        # the metric: a photograph against its kept reference, and one odd pair
        dict(name="score_4096x3072", kind="score", width=4096, height=3072),
        dict(name="pair_1023x767", kind="pair", width=1023, height=767),
        # the cover search of one photograph
        dict(name="select_1536x1024_rgb8", kind="select", width=1536, height=1024, bits=8,
             gaborish=True, scale=40000),
        # a gallery page of small streams to 8-bit pixels
        dict(name="decode_48_srgb8", kind="decode", streams=48, precision="fp32"),
    ]


def _draw_size(rng, lo: int, hi: int) -> dict:
    """Width and height of an area spread over its logarithm in [lo, hi]."""
    area = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    aspect = math.exp(rng.uniform(math.log(0.5), math.log(2.0)))
    width = max(16, int(math.sqrt(area * aspect)))
    return dict(width=width, height=max(16, int(area / width)))


def draw(rng) -> dict:
    kind = rng.choice(["probe", "probe", "sweep", "encode", "render", "score", "pair", "select",
                       "decode"])
    precision = rng.choice(["fp32", "fp32", "bf16x6", "bf16x3"])
    bits = rng.choice([8, 8, 12, 16])
    scale = int(math.exp(rng.uniform(math.log(16000), math.log(120000))))
    gaborish, epf = rng.choice([(True, 3), (True, 2), (True, 1), (False, 0), (False, 2)])
    if kind == "probe":
        return dict(_draw_size(rng, 1024, 1 << 22), kind=kind, bits=bits, precision=precision,
                    gaborish=gaborish, epf=epf, scale=scale)
    if kind == "sweep":
        return dict(_draw_size(rng, 1 << 12, 1 << 20), kind=kind, frames=rng.randint(1, 8),
                    bits=rng.choice([8, 16]), precision=precision, lanes=rng.choice([4, 8]))
    if kind == "encode":
        return dict(_draw_size(rng, 1 << 12, 3 << 22), kind=kind, bits=bits, precision=precision,
                    gaborish=gaborish, scale=scale)
    if kind == "render":
        return dict(_draw_size(rng, 1 << 12, 1 << 21), kind=kind, bits=bits, precision=precision,
                    gaborish=gaborish, epf=epf, scale=scale, out=rng.choice(["srgb8", "linear"]))
    if kind in ("score", "pair"):
        return dict(_draw_size(rng, 1 << 10, 3 << 22 if kind == "score" else 1 << 21), kind=kind)
    if kind == "select":
        return dict(_draw_size(rng, 1 << 12, 1 << 22), kind=kind, bits=bits, gaborish=gaborish,
                    scale=scale)
    return dict(kind="decode", streams=rng.randint(4, 48), precision=precision)


# ---- inputs -----------------------------------------------------------------

def _generator(seed: int, salt: int = 0) -> torch.Generator:
    g = torch.Generator(device="cuda")
    g.manual_seed((int(seed) * 1_000_003 + salt) & 0x7FFFFFFF)
    return g


def _image(width: int, height: int, bits: int, seed: int, salt: int = 0) -> torch.Tensor:
    """A photograph-like frame: [H, W, 3] code points (uint8, or int32 below
    2^bits).  Low sinusoids, noise with a 1/f spectrum and flat rectangles."""
    g = _generator(seed, salt)
    rand = lambda *s: torch.rand(*s, generator=g, device="cuda")  # noqa: E731
    yy = torch.arange(height, device="cuda", dtype=torch.float32)[:, None]
    xx = torch.arange(width, device="cuda", dtype=torch.float32)[None, :]
    fy = torch.fft.fftfreq(height, device="cuda")[:, None]
    fx = torch.fft.rfftfreq(width, device="cuda")[None, :]
    radius = torch.sqrt(fx * fx + fy * fy)
    shaping = torch.where(radius > 0, 1.0 / radius.clamp_min(1e-9), torch.zeros_like(radius))
    planes = []
    p = rand(3, 4, 4)
    for c in range(3):
        acc = torch.full((height, width), 128.0, device="cuda")
        for i in range(4):
            k = 2.0 * math.pi / (32.0 + 224.0 * p[c, i, 0])
            theta, phase = math.pi * p[c, i, 1], 2.0 * math.pi * p[c, i, 2]
            acc += (15.0 + 25.0 * p[c, i, 3]) * torch.sin(
                k * (torch.cos(theta) * xx + torch.sin(theta) * yy) + phase)
        white = torch.randn(height, width, generator=g, device="cuda")
        noise = torch.fft.irfft2(torch.fft.rfft2(white) * shaping, s=(height, width))
        acc += noise * (12.0 / noise.std().clamp_min(1e-6))
        planes.append(acc)
    out = torch.stack(planes, 2)
    r = rand(6, 7).cpu().numpy()
    for a in r:
        rw, rh = int(width * (0.06 + 0.27 * a[0])) + 1, int(height * (0.06 + 0.27 * a[1])) + 1
        x0, y0 = int((width - rw) * a[2]), int((height - rh) * a[3])
        out[y0:y0 + rh, x0:x0 + rw] = torch.tensor([255.0 * float(v) for v in a[4:7]],
                                                   device="cuda")
    top = (1 << bits) - 1
    codes = torch.clamp(torch.round(out * (top / 255.0)), 0, top)
    return codes.to(torch.uint8 if bits == 8 else torch.int32).contiguous()


def _as_input(codes: torch.Tensor, bits: int) -> torch.Tensor:
    """The code points as the package reads them: bytes, or 16-bit words."""
    return codes if bits == 8 else codes.to(torch.int16).contiguous()


def _linear(codes: torch.Tensor, bits: int) -> torch.Tensor:
    """The code points' linear light, float32 [3, H, W]."""
    v = codes.permute(2, 0, 1).to(torch.float64) / ((1 << bits) - 1)
    lin = torch.where(v <= 0.04045, v / 12.92, ((v + 0.055) / 1.055) ** 2.4)
    return lin.to(torch.float32).contiguous()


def _compressed(codes: torch.Tensor, step: float) -> torch.Tensor:
    """The 8-bit frame after 8x8 block-transform quantization: the artifacts
    the metric is used on."""
    h, w, _ = codes.shape
    x = codes.permute(2, 0, 1).to(torch.float32)
    x = torch.nn.functional.pad(x, (0, -w % 8, 0, -h % 8), mode="replicate")
    hh, ww = x.shape[1:]
    d = torch.tensor([[math.cos(math.pi * (2 * i + 1) * u / 16) * (0.5 if u else math.sqrt(0.125))
                       for i in range(8)] for u in range(8)], device="cuda")
    b = x.reshape(3, hh // 8, 8, ww // 8, 8).permute(0, 1, 3, 2, 4)
    f = d @ b @ d.T
    u = torch.arange(8, device="cuda", dtype=torch.float32)
    q = step * (1.0 + 0.35 * (u[:, None] + u[None, :]))
    b = d.T @ (torch.round(f / q) * q) @ d
    x = b.permute(0, 1, 3, 2, 4).reshape(3, hh, ww)[:, :h, :w]
    return torch.clamp(torch.round(x), 0, 255).permute(1, 2, 0).to(torch.uint8)


_CONTEXT = None


def _context() -> "jg.Context":
    """The context a program keeps for all its calls."""
    global _CONTEXT
    if _CONTEXT is None:
        _CONTEXT = jg.Context(0)
    return _CONTEXT


def _request(case: dict, scale: int | None = None) -> "jg.EncodeRequest":
    return jg.EncodeRequest.with_global_scale(
        scale or case.get("scale", 40000), gaborish=case.get("gaborish", True),
        epf_iters=case.get("epf", 3), precision=case.get("precision", "fp32"))


def _layout(ctx, width: int, height: int, rgb: torch.Tensor, bits: int, req) -> "jg.Layout":
    """The encoder's own cover at the request's quantizer."""
    bmap = torch.zeros(((height + 7) // 8, (width + 7) // 8), dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    jg.select_blocks_device(ctx, width, height, rgb.data_ptr(), bits, req, bmap.data_ptr())
    ctx.synchronize()
    return jg.Layout(ctx, width, height, bmap.cpu().numpy(), 1, 7)


def _reference(ctx, linear: torch.Tensor) -> "jg.PrecomputedReference":
    torch.cuda.synchronize()
    ref = jg.PrecomputedReference(ctx, device_ptr=linear.data_ptr(), width=linear.shape[2],
                                  height=linear.shape[1])
    ctx.synchronize()
    return ref


def _plan_buffers(layout) -> dict:
    z = lambda t, *s: torch.zeros(*s, dtype=t, device="cuda")  # noqa: E731
    return dict(qcoeff=z(torch.int32, 3, 8 * layout.bh, 8 * layout.bw),
                lf=z(torch.int32, 3, layout.bh, layout.bw),
                cfl_x=z(torch.int8, layout.th, layout.tw),
                cfl_b=z(torch.int8, layout.th, layout.tw))


def _plan_struct(plan: dict, factors=(128, 128)) -> PlanStruct:
    s = PlanStruct()
    for k in ("qcoeff", "lf", "cfl_x", "cfl_b"):
        setattr(s, k, plan[k].data_ptr())
    s.lf_factors[0], s.lf_factors[1] = int(factors[0]), int(factors[1])
    return s


def _encode_into(ctx, layout, rgb, bits, params, plan, struct) -> None:
    ctx.check(ctx.lib.jpxlg_encode_transform(ctx.handle, layout.handle,
                                             C.c_void_p(rgb.data_ptr()), bits, C.byref(params),
                                             C.byref(struct), jg.MEM_DEVICE))


def _sweep_sizes(case: dict) -> list:
    """Uneven frame sizes up to the case's width x height."""
    n, w, h = case["frames"], case["width"], case["height"]
    frac = lambda v: v - math.floor(v)  # noqa: E731
    return [(max(16, int(w * (0.2 + 0.8 * frac(0.618034 * (i + 1))))),
             max(16, int(h * (0.2 + 0.8 * frac(0.414214 * (i + 1)))))) for i in range(n)]


SWEEP_SCALES = (16000, 22000, 30000, 40000, 52000, 68000, 90000, 120000)


def prepare(case: dict, seed: int) -> dict:
    kind, ctx = case["kind"], _context()
    st = dict(case=case, kind=kind, ctx=ctx)
    if kind in ("probe", "encode", "render", "select"):
        w, h, bits = case["width"], case["height"], case["bits"]
        codes = _image(w, h, bits, seed)
        rgb = _as_input(codes, bits)
        req = _request(case)
        st.update(rgb=rgb, req=req, bits=bits, width=w, height=h)
        if kind == "select":
            st["map"] = torch.zeros(((h + 7) // 8, (w + 7) // 8), dtype=torch.uint8,
                                    device="cuda")
            return st
        layout = _layout(ctx, w, h, rgb, bits, req)
        st["layout"] = layout
        if kind == "probe":
            st["ref"] = _reference(ctx, _linear(codes, bits))
            st["score"] = torch.zeros(1, dtype=torch.float64, device="cuda")
            return st
        params, plan = req._struct(), _plan_buffers(layout)
        st.update(params=params, plan=plan, struct=_plan_struct(plan))
        if kind == "render":
            torch.cuda.synchronize()
            _encode_into(ctx, layout, rgb, bits, params, plan, st["struct"])
            st["out"] = (torch.zeros(h, w, 3, dtype=torch.uint8, device="cuda")
                         if case["out"] == "srgb8"
                         else torch.zeros(3, h, w, dtype=torch.float32, device="cuda"))
        return st
    if kind == "sweep":
        items, keep = [], []
        for i, (w, h) in enumerate(_sweep_sizes(case)):
            codes = _image(w, h, case["bits"], seed, salt=7919 * (i + 1))
            rgb = _as_input(codes, case["bits"])
            ref = _reference(ctx, _linear(codes, case["bits"]))
            keep.append((rgb, ref))
            for gs in SWEEP_SCALES:
                req = _request(case, gs)
                layout = _layout(ctx, w, h, rgb, case["bits"], req)
                items.append(jg.BatchItem(layout, ref, rgb.data_ptr(), case["bits"], req))
        st.update(keep=keep, items=items)
        st["batch"] = jg.BatchProbe(ctx, items, case["lanes"])
        st["scores"] = torch.zeros(len(items), dtype=torch.float64, device="cuda")
        return st
    if kind in ("score", "pair"):
        w, h = case["width"], case["height"]
        codes = _image(w, h, 8, seed)
        step = 4.0 + 20.0 * float(torch.rand(1, generator=_generator(seed, 1), device="cuda"))
        st.update(source=_linear(codes, 8), cand=_linear(_compressed(codes, step), 8), width=w,
                  height=h)
        if kind == "score":
            st["ref"] = _reference(ctx, st["source"])
            z = lambda n: torch.zeros(n, dtype=torch.float64, device="cuda")  # noqa: E731
            st.update(score=z(1), raw=z(1), terms=z(18 * len(_scales(w, h))))
        else:
            torch.cuda.synchronize()
        return st
    # decode: the seed picks the grey streams
    pick = np.random.default_rng(seed).integers(0, len(GREY_STREAMS), case["streams"])
    names = [RGB_STREAMS.get(i % STREAM_SLOTS, GREY_STREAMS[p]) for i, p in enumerate(pick)]
    datas = [(STREAMS / (n + ".jxl")).read_bytes() for n in names]
    st["opened"] = jg.open_codestreams(datas)
    st["batch"] = jg.DecodeBatch(ctx, st["opened"], "srgb8", precision=case["precision"])
    return st


def run(st: dict):
    kind, ctx = st["kind"], st["ctx"]
    if kind == "probe":
        ctx.probe_device(st["layout"], st["ref"], st["rgb"].data_ptr(), st["bits"], st["req"],
                         st["score"].data_ptr())
        return st["score"]
    if kind == "sweep":
        st["batch"].run_device(st["scores"].data_ptr())
        return st["scores"]
    if kind == "encode":
        s = st["struct"]
        _encode_into(ctx, st["layout"], st["rgb"], st["bits"], st["params"], st["plan"], s)
        return dict(st["plan"], lf_factors=[int(s.lf_factors[0]), int(s.lf_factors[1])])
    if kind == "render":
        out = jg.OUT_SRGB8 if st["case"]["out"] == "srgb8" else jg.OUT_LINEAR
        ctx.check(ctx.lib.jpxlg_reconstruct(ctx.handle, st["layout"].handle, C.byref(st["struct"]),
                                            C.byref(st["params"]), out, st["bits"],
                                            C.c_void_p(st["out"].data_ptr()), jg.MEM_DEVICE))
        return st["out"]
    if kind == "score":
        ctx.check(ctx.lib.jpxlg_ssim2_score(
            ctx.handle, st["ref"].handle, C.c_void_p(st["cand"].data_ptr()), jg.MEM_DEVICE,
            C.cast(st["score"].data_ptr(), C.POINTER(C.c_double)),
            C.cast(st["raw"].data_ptr(), C.POINTER(C.c_double)),
            C.c_void_p(st["terms"].data_ptr())))
        return dict(score=st["score"], raw=st["raw"], terms=st["terms"])
    if kind == "pair":
        out = C.c_double()
        ctx.check(ctx.lib.jpxlg_score_pair(
            ctx.handle, C.c_void_p(st["source"].data_ptr()), C.c_void_p(st["cand"].data_ptr()),
            st["width"], st["height"], jg.MEM_DEVICE, C.byref(out)))
        return out.value
    if kind == "select":
        jg.select_blocks_device(ctx, st["width"], st["height"], st["rgb"].data_ptr(), st["bits"],
                                st["req"], st["map"].data_ptr())
        return st["map"]
    return st["batch"].run()


# ---- the work that a pass cannot do without ---------------------------------
# Bytes count each input read and each output written once (the coefficient
# image and the metric's reference planes are inputs or outputs where the
# call has them).  Operations per pixel, f32: opsin mix and cube roots 60;
# inverse Gaborish 12 x 14 x 3; one separable DCT of three channels 60;
# quantizer 45; CfL's eight candidates 120; Gaborish 54; EPF steps 400, 140
# and 70; opsin inverse 40; the metric per pyramid pixel 60 (XYB) + 18 x 13
# (nine quantities, two passes of a symmetric nine-tap sum) + 6 + 105.

def _scales(w: int, h: int) -> list:
    """The metric's scales: halved (rounded up) while the last is at least 8x8."""
    out = [(w, h)]
    while len(out) < 6 and min(out[-1]) >= 8:
        out.append(((out[-1][0] + 1) // 2, (out[-1][1] + 1) // 2))
    return out


def _encode_flops(gaborish: bool) -> float:
    return 60 + (504 if gaborish else 0) + 60 + 45 + 120


def _render_flops(gaborish: bool, epf: int) -> float:
    return 60 + 15 + (54 if gaborish else 0) + (0, 140, 210, 610)[epf] + 40


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "decode":
        px = case["streams"] * STREAM_PIXELS
        return dict(bytes=px * (12.2 + 3.0), flops=px * _render_flops(True, 1))
    if kind == "sweep":
        b = f = 0.0
        for w, h in _sweep_sizes(case):
            one = work(dict(case, kind="probe", width=w, height=h, gaborish=True, epf=3))
            b, f = b + len(SWEEP_SCALES) * one["bytes"], f + len(SWEEP_SCALES) * one["flops"]
        return dict(bytes=b, flops=f)
    w, h = case["width"], case["height"]
    px = w * h
    pyramid = sum(a * b for a, b in _scales(w, h))
    if kind == "score":
        return dict(bytes=12.0 * px + 36.0 * pyramid, flops=405.0 * pyramid)
    if kind == "pair":
        return dict(bytes=24.0 * px, flops=(60 + 6 * 13 * 2 + 405.0) * pyramid)
    src = px * (3.0 if case["bits"] == 8 else 6.0)
    gab, epf = case["gaborish"], case.get("epf", 0)
    if kind == "select":
        return dict(bytes=src + px / 64, flops=px * (60 + (504 if gab else 0) + 3 * (60 + 60)))
    if kind == "encode":
        return dict(bytes=src + 12.2 * px, flops=px * _encode_flops(gab))
    if kind == "render":
        return dict(bytes=px * (12.2 + (3.0 if case["out"] == "srgb8" else 12.0)),
                    flops=px * _render_flops(gab, epf))
    return dict(bytes=src + 36.0 * pyramid,
                flops=px * (_encode_flops(gab) + _render_flops(gab, epf)) + 405.0 * pyramid)


# ---- 64-bit results ----------------------------------------------------------

MIX = ((0.3, 0.622, 0.078), (0.23, 0.692, 0.078), (0.2434227, 0.2047674, 0.5518099))
OPSIN_INVERSE = ((11.031567, -9.866944, -0.16462299), (-3.2541474, 4.4187705, -0.16462299),
                 (-3.6588513, 2.712923, 1.9459282))
# SSIMULACRA2's weights: channel, scale, norm (mean, fourth power), map.
METRIC_WEIGHTS = (
    0.0, 0.0007376606707406586, 0.0, 0.0, 0.0007793481682867309, 0.0, 0.0, 0.0004371155730107379,
    0.0, 1.1041726426657346, 0.00066284834129271, 0.00015231632783718752, 0.0,
    0.0016406437456599754, 0.0, 1.8422455520539298, 11.441172603757666, 0.0,
    0.0007989109436015163, 0.000176816438078653, 0.0, 1.8787594979546387, 10.94906990605142, 0.0,
    0.0007289346991508072, 0.9677937080626833, 0.0, 0.00014003424285435884, 0.9981766977854967,
    0.00031949755934435053, 0.0004550992113792063, 0.0, 0.0, 0.0013648766163243398, 0.0, 0.0, 0.0,
    0.0, 0.0, 7.466890328078848, 0.0, 17.445833984131262, 0.0006235601634041466, 0.0, 0.0,
    6.683678146179332, 0.00037724407979611296, 1.027889937768264, 225.20515300849274, 0.0, 0.0,
    19.213238186143016, 0.0011401524586618361, 0.001237755635509985, 176.39317598450694, 0.0, 0.0,
    24.43300999870476, 0.28520802612117757, 0.0004485436923833408, 0.0, 0.0, 0.0,
    34.77906344483772, 44.835625328877896, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0,
    0.0008680556573291698, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0005313191874358747, 0.0,
    0.00016533814161379112, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0004179171803251336,
    0.0017290828234722833, 0.0, 0.0020827005846636437, 0.0, 0.0, 8.826982764996862,
    23.19243343998926, 0.0, 95.1080498811086, 0.9863978034400682, 0.9834382792465353,
    0.0012286405048278493, 171.2667255897307, 0.9807858872435379, 0.0, 0.0, 0.0,
    0.0005130064588990679, 0.0, 0.00010854057858411537)
RESONATOR_IN = (0.05529523572608661, -0.05883668702694998, 0.012955819110517063)
RESONATOR_PREV = (1.902113032590307, 1.1755705045849463, 1.2246467991473532e-16)


def _cbrt(x: torch.Tensor) -> torch.Tensor:
    y = torch.sign(x) * torch.abs(x) ** (1.0 / 3.0)
    return torch.where(y == 0, y, y - (y * y * y - x) / (3.0 * y * y).clamp_min(1e-300))


def _positive_xyb(lin: torch.Tensor) -> torch.Tensor:
    g = [_cbrt(m[0] * lin[0] + m[1] * lin[1] + m[2] * lin[2] + 0.0037930734) - 0.1559542
         for m in MIX]
    x, y = 0.5 * (g[0] - g[1]), 0.5 * (g[0] + g[1])
    return torch.stack([14.0 * x + 0.42, y + 0.01, g[2] - y + 0.55])


def _blur_taps() -> list:
    """The recursive Gaussian's response at distances 0..4 (finite: the
    resonators cancel beyond)."""
    taps = []
    for d in range(5):
        prev, prev2, out = [0.0] * 3, [0.0] * 3, 0.0
        for j in range(16 + d + 1):
            s = (1.0 if j + 4 == 16 else 0.0) + (1.0 if j - 6 == 16 else 0.0)
            o = [s * RESONATOR_IN[k] + RESONATOR_PREV[k] * prev[k] - prev2[k] for k in range(3)]
            prev2, prev, out = prev, o, (o[0] + o[1]) + o[2]
        taps.append(out)
    return taps


def _blur(x: torch.Tensor) -> torch.Tensor:
    taps = _blur_taps()
    for dim in (2, 1):
        pad = (4, 4, 0, 0) if dim == 2 else (0, 0, 4, 4)
        n, p = x.shape[dim], torch.nn.functional.pad(x, pad)
        x = taps[0] * p.narrow(dim, 4, n) + sum(
            taps[d] * (p.narrow(dim, 4 - d, n) + p.narrow(dim, 4 + d, n)) for d in range(1, 5))
    return x


def _downscale(x: torch.Tensor) -> torch.Tensor:
    h, w = x.shape[1:]
    x = torch.nn.functional.pad(x[None], (0, w % 2, 0, h % 2), mode="replicate")[0]
    return (x[:, ::2, ::2] + x[:, ::2, 1::2] + x[:, 1::2, ::2] + x[:, 1::2, 1::2]) * 0.25


def _ssimulacra2(source: torch.Tensor, cand: torch.Tensor) -> dict:
    a, b = source.to(torch.float64), cand.to(torch.float64)
    terms = []
    for s in range(6):
        if s:
            if min(a.shape[1:]) < 8:
                break
            a, b = _downscale(a), _downscale(b)
        xa, xb = _positive_xyb(a), _positive_xyb(b)
        m1, m2 = _blur(xa), _blur(xb)
        s11, s22, s12 = _blur(xa * xa), _blur(xb * xb), _blur(xa * xb)
        d = torch.clamp_min(
            1.0 - ((1.0 - (m1 - m2) ** 2) * (2.0 * (s12 - m1 * m2) + 0.0009))
            / ((s11 - m1 * m1) + (s22 - m2 * m2) + 0.0009), 0.0)
        r = (1.0 + torch.abs(xb - m2)) / (1.0 + torch.abs(xa - m1)) - 1.0
        maps = (d, torch.clamp_min(r, 0.0), torch.clamp_min(-r, 0.0))
        mean = [m.mean((1, 2)) for m in maps]
        four = [(m ** 4).mean((1, 2)) ** 0.25 for m in maps]
        terms.append(torch.stack(mean + four, 1))  # [channel, 6]
    t = torch.stack(terms)  # [scale, channel, 6]
    flat = t.permute(1, 0, 2).reshape(-1).cpu().tolist()
    err = math.fsum(w * abs(v) for w, v in zip(METRIC_WEIGHTS, flat))
    e = err * 0.9562382616834844
    e = 6.248496625763138e-5 * e ** 3 + 2.326765642916932 * e - 0.020884521182843837 * e * e
    score = 100.0 - 10.0 * e ** 0.6276336467831387 if e > 0.0 else 100.0
    return dict(score=score, raw=err, terms=t.reshape(-1))


# DCT8, DCT16 and DCT32 dequantization bands per channel (X, Y, B).
BANDS = {
    8: ((3150.0, 0.0, -0.4, -0.4, -0.4, -2.0), (560.0, 0.0, -0.3, -0.3, -0.3, -0.3),
        (512.0, -2.0, -1.0, 0.0, -1.0, -2.0)),
    16: ((8996.8725711814115328, -1.3000777393353804, -0.49424529824571225, -0.439093774457103443,
          -0.6350101832695744, -0.90177264050827612, -1.6162099239887414),
         (3191.48366296844234752, -0.67424582104194355, -0.80745813428471001,
          -0.44925837484843441, -0.35865440981033403, -0.31322389111877305,
          -0.37615025315725483),
         (1157.50408145487200256, -2.0531423165804414, -1.4, -0.50687130033378396,
          -0.42708730624733904, -1.4856834539296244, -4.9209142884401604)),
    32: ((15718.40830982518931456, -1.025, -0.98, -0.9012, -0.4, -0.48819395464, -0.421064,
          -0.27),
         (7305.7636810695983104, -0.8041958212306401, -0.7633036457487539, -0.55660379990111464,
          -0.49785304658857626, -0.43699592683512467, -0.40180866526242109,
          -0.27321683125358037),
         (3803.53173721215041536, -3.060733579805728, -2.0413270132490346, -2.0235650159727417,
          -0.5495389509954993, -0.4, -0.4, -0.3)),
}


def _dequant_matrix(n: int, c: int) -> torch.Tensor:
    p = BANDS[n][c]
    bands = [p[0]]
    for v in p[1:]:
        bands.append(bands[-1] * (1.0 + v if v > 0.0 else 1.0 / (1.0 - v)))
    m = torch.zeros(n, n, dtype=torch.float64)
    for y in range(n):
        for x in range(n):
            pos = math.hypot(x / (n - 1), y / (n - 1)) * (len(p) - 1) / (math.sqrt(2.0) + 1e-6)
            i = int(pos)
            m[y, x] = 1.0 / (bands[i] * (bands[i + 1] / bands[i]) ** (pos - i))
    return m.cuda()


def _inverse_basis(n: int) -> torch.Tensor:
    """I[i, u]: samples from coefficients whose (0, 0) is the mean."""
    i = torch.arange(n, dtype=torch.float64)[:, None]
    u = torch.arange(n, dtype=torch.float64)[None, :]
    m = math.sqrt(2.0) * torch.cos(math.pi * (2.0 * i + 1.0) * u / (2.0 * n))
    m[:, 0] = 1.0
    return m.cuda()


def _mirrored(x: torch.Tensor, r: int) -> torch.Tensor:
    """Planes with r mirrored samples (edge repeated) on every side."""
    def index(n):
        i = torch.arange(-r, n + r, device="cuda") % (2 * n)
        return torch.where(i < n, i, 2 * n - 1 - i)
    return x[:, index(x.shape[1])][:, :, index(x.shape[2])]


def _gaborish(x: torch.Tensor) -> torch.Tensor:
    w1, w2 = 0.115169525, 0.061248592
    h, w = x.shape[1:]
    p = _mirrored(x, 1)
    at = lambda dy, dx: p[:, 1 + dy:1 + dy + h, 1 + dx:1 + dx + w]  # noqa: E731
    edge = at(-1, 0) + at(1, 0) + at(0, -1) + at(0, 1)
    corner = at(-1, -1) + at(-1, 1) + at(1, -1) + at(1, 1)
    return (at(0, 0) + w1 * edge + w2 * corner) / (1.0 + 4.0 * w1 + 4.0 * w2)


CROSS = ((0, 0), (-1, 0), (1, 0), (0, -1), (0, 1))
DIAMOND = CROSS + ((1, -1), (1, 1), (-1, 1), (-1, -1), (-2, 0), (2, 0), (0, 2), (0, -2))


def _epf_step(step: int, x: torch.Tensor, sigma: torch.Tensor) -> torch.Tensor:
    h, w = x.shape[1:]
    p = _mirrored(x, 3)
    at = lambda dy, dx: p[:, 3 + dy:3 + dy + h, 3 + dx:3 + dx + w]  # noqa: E731
    gain = torch.tensor([40.0, 5.0, 3.5], dtype=torch.float64, device="cuda")[:, None, None]
    inv = 1.65 * (0.9, 1.0, 6.5)[step] * 4.0 * (1.0 - math.sqrt(0.5)) / sigma
    yy = torch.arange(h, device="cuda")[:, None] % 8
    xx = torch.arange(w, device="cuda")[None, :] % 8
    border = (yy == 0) | (yy == 7) | (xx == 0) | (xx == 7)
    pos = torch.where(border, torch.full((), 2.0 / 3.0, dtype=torch.float64, device="cuda"),
                      torch.ones((), dtype=torch.float64, device="cuda"))
    total, acc = torch.zeros_like(sigma), torch.zeros_like(x)
    for kx, ky in (DIAMOND if step == 0 else CROSS):
        d = torch.zeros_like(sigma)
        for ix, iy in (CROSS if step < 2 else ((0, 0),)):
            d += (gain * torch.abs(at(iy, ix) - at(ky + iy, kx + ix))).sum(0)
        wt = torch.clamp_min(1.0 - pos * d * inv, 0.0)
        total += wt
        acc += wt * at(ky, kx)
    return torch.where(sigma < 0.3, x, acc / total)


def _rendered(st: dict) -> torch.Tensor:
    """The plan's linear planes: dequantize, HF and LF chroma from luma,
    inverse DCTs of the square varblocks, Gaborish, EPF, opsin inverse."""
    case, layout, plan = st["case"], st["layout"], st["plan"]
    w, h, f64 = st["width"], st["height"], torch.float64
    gs, quant_lf = case["scale"], st["req"].quant_lf
    bh, bw = layout.bh, layout.bw
    fx, fb = (int(st["struct"].lf_factors[i]) - 128 for i in range(2))
    lf = plan["lf"].to(f64) * torch.tensor(
        [65536.0 * v / 128.0 / (gs * quant_lf) for v in (1 / 32, 1 / 4, 1 / 2)], dtype=f64,
        device="cuda")[:, None, None]
    lf = torch.stack([lf[0] + fx / 84.0 * lf[1], lf[1], lf[2] + (1.0 + fb / 84.0) * lf[1]])
    q = plan["qcoeff"].to(f64)
    bias = 1.0 - torch.tensor([0.054650073, 0.0700545, 0.049935103], dtype=f64,
                              device="cuda")[:, None, None]
    big = torch.where(q.abs() > 1, q, torch.full_like(q, 2.0))
    q = torch.where(q.abs() > 1, big - 0.145 / big, q * bias) * (65536.0 / gs)
    tile = lambda t: t.to(f64).repeat_interleave(64, 0).repeat_interleave(  # noqa: E731
        64, 1)[:8 * bh, :8 * bw]
    kx, kb = tile(plan["cfl_x"]) / 84.0, 1.0 + tile(plan["cfl_b"]) / 84.0
    planes = torch.zeros(3, 8 * bh, 8 * bw, dtype=f64, device="cuda")
    bmap = torch.from_numpy(layout.block_map).cuda()
    for sel, n in ((0, 8), (4, 16), (5, 32)):
        by, bx = torch.nonzero(bmap == (sel | 0x80), as_tuple=True)
        if not len(by):
            continue
        k = n // 8
        r = torch.arange(n, device="cuda")
        ys, xs = (by * 8)[:, None, None] + r[None, :, None], (bx * 8)[:, None, None] + r
        m = torch.stack([_dequant_matrix(n, c) for c in range(3)])[:, None]
        co = q[:, ys, xs] * m
        co = torch.stack([co[0] + kx[ys, xs] * co[1], co[1], co[2] + kb[ys, xs] * co[1]])
        # the coefficient matrix holds horizontal frequencies down its rows
        rr = torch.arange(k, device="cuda")
        rect = lf[:, by[:, None, None] + rr[None, :, None], bx[:, None, None] + rr]
        fwd = _inverse_basis(k).T / k
        u = torch.arange(k, dtype=f64)
        sf = (1.0 / (torch.cos(u * math.pi / (2 * n)) * torch.cos(u * math.pi / n)
                     * torch.cos(2.0 * u * math.pi / n))).cuda()
        llf = (fwd @ rect @ fwd.T).transpose(-1, -2) * sf[:, None] * sf[None, :]
        co[..., :k, :k] = llf
        inv = _inverse_basis(n)
        planes[:, ys, xs] = inv @ co.transpose(-1, -2) @ inv.T
    planes = planes[:, :h, :w]
    sigma = torch.full((h, w), 65536.0 / gs * 0.46, dtype=f64, device="cuda")
    if case["gaborish"]:
        planes = _gaborish(planes)
    for step in ((), (1,), (1, 2), (0, 1, 2))[case["epf"]]:
        planes = _epf_step(step, planes, sigma)
    root = -(0.0037930733 ** (1.0 / 3.0))
    g = torch.stack([planes[1] + planes[0], planes[1] - planes[0], planes[2]]) - root
    mix = g ** 3 - 0.0037930733
    return torch.stack([m[0] * mix[0] + m[1] * mix[1] + m[2] * mix[2] for m in OPSIN_INVERSE])


def exact(case: dict, seed: int):
    """Whole numbers (plans, covers, 8-bit pixels) have no 64-bit value, nor
    has the score of a probe, which follows from its plan's integers."""
    kind = case["kind"]
    if kind == "render" and case["out"] == "linear":
        return _rendered(prepare(case, seed))
    if kind in ("score", "pair"):
        st = prepare(case, seed)
        r = _ssimulacra2(st["source"], st["cand"])
        if kind == "pair":
            return r["score"]
        one = lambda v: torch.tensor([v], dtype=torch.float64, device="cuda")  # noqa: E731
        return dict(score=one(r["score"]), raw=one(r["raw"]), terms=r["terms"])
    return None
