"""Gaborish and EPF at the edges of their tiles, bit for bit against the
restatement's XYB planes.

Widths around the EPF's 60 and 64 pixel columns and the 16-byte rows that
the tiles and Gaborish load at once, heights around its 6 and 8, 14 and 16, 22
and 24 rows (runs of two, four and six rows by the frame's size) and
Gaborish's runs of eight; every step count, sharpness 0 .. 7 (blocks that
are copied among them) and uneven hf_mul.
"""
import numpy as np
import pytest

import jpxl_gb300 as jg
from jpxl_gb300 import synth

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (3, 2), (8, 8), (60, 22), (61, 23), (64, 24), (65, 25), (68, 45), (72, 50),
         (123, 44), (124, 47), (128, 96), (131, 73), (192, 71), (200, 120), (252, 68),
         (240, 362), (253, 378), (601, 425), (640, 462)]


@pytest.mark.parametrize("epf", [1, 2, 3])
@pytest.mark.parametrize("w,h", SIZES)
def test_filters_at_tile_edges(ctx, oracle, w, h, epf):
    rng = np.random.default_rng(1000 * epf + w * 31 + h)
    bw, bh = (w + 7) // 8, (h + 7) // 8
    bmap = synth.fixed_dct8_map(w, h)
    q = (rng.integers(-6, 7, (3, bh * 8, bw * 8)) * (rng.random((3, bh * 8, bw * 8)) < 0.2))
    plan = {"qcoeff": q.astype(np.int32),
            "lf": rng.integers(-40, 400, (3, bh, bw)).astype(np.int32),
            "cfl_x": np.zeros(((bh + 7) // 8, (bw + 7) // 8), np.int8),
            "cfl_b": np.zeros(((bh + 7) // 8, (bw + 7) // 8), np.int8), "lf_factors": (128, 128)}
    hf = rng.integers(1, 6, bmap.shape).astype(np.uint32)
    sh = rng.integers(0, 8, bmap.shape).astype(np.uint8)
    layout = jg.Layout(ctx, w, h, bmap, hf, sh)
    p = jg.Plan(plan["qcoeff"], plan["lf"], plan["cfl_x"], plan["cfl_b"], plan["lf_factors"])
    gab = bool((w + h) % 3)
    req = jg.EncodeRequest(global_scale=9000, quant_lf=8, gaborish=gab, epf_iters=epf)
    got = jg.PlanRenderer(ctx).render(layout, p, req, out="xyb")
    rc, want = oracle.reconstruct(w, h, bmap, hf, sh, plan, global_scale=9000, quant_lf=8,
                                  gaborish=gab, epf_iters=epf, out_kind=0)
    assert rc == 0
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
