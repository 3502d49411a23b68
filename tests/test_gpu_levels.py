"""The colour output's levels and the cube roots, bit for bit against the
restatement: rendered XYB that spreads over dark, bright and out-of-range
light (negative and above one, where a level clamps and a cube root leaves
its short path), at 8-bit sRGB and at depths from 1 to 16 bits, and the XYB
of 8-bit frames."""
import numpy as np
import pytest

import jpxl_gb300 as jg
from jpxl_gb300 import synth

pytestmark = pytest.mark.gpu


def _plan(w, h, seed):
    rng = np.random.default_rng(seed)
    bw, bh = (w + 7) // 8, (h + 7) // 8
    q = rng.integers(-4, 5, (3, bh * 8, bw * 8)) * (rng.random((3, bh * 8, bw * 8)) < 0.1)
    # Y of 0 .. 0.85 in steps of 0.0013, X about zero, B beside Y: light from
    # dark to about one, and what the HF adds on either side
    lf = np.stack([rng.integers(-60, 61, (bh, bw)), rng.integers(0, 640, (bh, bw)),
                   rng.integers(0, 320, (bh, bw))])
    return {"qcoeff": q.astype(np.int32), "lf": lf.astype(np.int32),
            "cfl_x": np.zeros(((bh + 7) // 8, (bw + 7) // 8), np.int8),
            "cfl_b": np.zeros(((bh + 7) // 8, (bw + 7) // 8), np.int8), "lf_factors": (128, 128)}


@pytest.mark.parametrize("out,bits", [("srgb8", 8), ("linear_at_depth", 1),
                                      ("linear_at_depth", 8), ("linear_at_depth", 9),
                                      ("linear_at_depth", 12), ("linear_at_depth", 16)])
def test_levels_of_light_in_and_out_of_range(ctx, oracle, out, bits):
    w, h = 173, 131
    plan = _plan(w, h, 40 + bits)
    bmap = synth.fixed_dct8_map(w, h)
    hf = np.ones(bmap.shape, np.uint32)
    sh = np.full(bmap.shape, 4, np.uint8)
    layout = jg.Layout(ctx, w, h, bmap, hf, sh)
    p = jg.Plan(plan["qcoeff"], plan["lf"], plan["cfl_x"], plan["cfl_b"], plan["lf_factors"])
    req = jg.EncodeRequest(global_scale=12000, quant_lf=8)
    lin = jg.PlanRenderer(ctx).render(layout, p, req, out="linear")
    assert lin.min() < -0.01 and lin.max() > 1.01 and np.median(np.abs(lin)) < 0.9
    got = jg.PlanRenderer(ctx).render(layout, p, req, out=out, bits=bits)
    rc, want = oracle.reconstruct(w, h, bmap, hf, sh, plan, global_scale=12000, quant_lf=8,
                                  out_kind=2 if out == "srgb8" else 3, bits=bits)
    assert rc == 0 and got.dtype == want.dtype
    assert np.array_equal(got.view(np.uint8), want.view(np.uint8))


def test_xyb_of_every_8bit_code_point(ctx, oracle):
    """Every code in every channel, beside mid and extreme neighbours."""
    codes = np.arange(256, dtype=np.uint8)
    cols = [np.stack(c, 1) for o in (0, 1, 128, 255)
            for c in ((codes, codes * 0 + o, codes[::-1]), (codes * 0 + o, codes, codes),
                      (codes[::-1], codes, codes * 0 + o), (codes, codes, codes))]
    rgb = np.ascontiguousarray(np.stack(cols, 0))
    h, w = rgb.shape[:2]
    bmap = synth.fixed_dct8_map(w, h)
    layout = jg.Layout(ctx, w, h, bmap)
    st = ctx.encode_stages(layout, rgb, jg.EncodeRequest(global_scale=30000))
    rc, ref = oracle.encode(rgb, bmap, np.ones(bmap.shape, np.uint32), global_scale=30000,
                            stages=True)
    assert rc == 0
    assert np.array_equal(st["xyb"].view(np.uint32), ref["xyb"].view(np.uint32))
