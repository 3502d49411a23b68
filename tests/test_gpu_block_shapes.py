"""Every block side of 8 to 32 but DCT8 itself, bit for bit against the
restatement: one block, odd numbers of them (a warp spans several narrow
blocks), and frames that cut the last blocks off anywhere."""
import numpy as np
import pytest

import jpxl_gb300 as jg
from jpxl_gb300 import synth

pytestmark = pytest.mark.gpu

CASES = [(n, cols, rows, cut) for n in (16, 32) for cols, rows in ((1, 1), (3, 1), (2, 2), (5, 3))
         for cut in (0, 1, 7)]


def _cover(n, cols, rows):
    m = synth.fixed_dct8_map(cols * n, rows * n)
    for by in range(rows):
        for bx in range(cols):
            synth.place(m, bx * n // 8, by * n // 8, synth.DCT16 if n == 16 else synth.DCT32)
    return m


@pytest.mark.parametrize("n,cols,rows,cut", CASES)
def test_square_blocks(ctx, oracle, n, cols, rows, cut):
    w, h = cols * n - cut, rows * n - (cut * 5) % 8
    bmap = _cover(n, cols, rows)
    rng = np.random.default_rng(n + 10 * cols + cut)
    rgb = rng.integers(0, 256, (h, w, 3)).astype(np.uint8)
    hf = rng.integers(1, 9, bmap.shape).astype(np.uint32)
    sh = rng.integers(0, 9, bmap.shape).astype(np.uint8)
    req = jg.EncodeRequest(global_scale=15000, gaborish=True, epf_iters=2)
    layout = jg.Layout(ctx, w, h, bmap, hf, sh)
    plan = ctx.encode_transform(layout, rgb, req)
    rc, ref = oracle.encode(rgb, bmap, hf, global_scale=15000, gaborish=True)
    assert rc == 0
    for k in ("qcoeff", "lf", "cfl_x", "cfl_b"):
        assert np.array_equal(getattr(plan, k), ref[k]), k
    got = jg.PlanRenderer(ctx).render(layout, plan, req, out="xyb")
    rc, want = oracle.reconstruct(w, h, bmap, hf, sh, ref, global_scale=15000, gaborish=True,
                                  epf_iters=2, out_kind=0)
    assert rc == 0
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))


RECTS = [s for s, rc in synth.SHAPES.items() if rc[0] != rc[1]]


@pytest.mark.parametrize("cut", [0, 3])
@pytest.mark.parametrize("cols,rows", [(1, 1), (3, 1), (2, 3)])
@pytest.mark.parametrize("sel", RECTS)
def test_rectangles(ctx, oracle, sel, cols, rows, cut):
    """Rectangles share the inverse kernel: counts that fill a block group and
    that leave places of it idle."""
    r, c = synth.SHAPES[sel]
    w, h = cols * c * 8 - cut, rows * r * 8 - (cut * 5) % 8
    bmap = synth.fixed_dct8_map(cols * c * 8, rows * r * 8)
    for by in range(rows):
        for bx in range(cols):
            synth.place(bmap, bx * c, by * r, sel)
    rng = np.random.default_rng(sel * 100 + cols * 10 + cut)
    bh, bw = bmap.shape
    q = rng.integers(-6, 7, (3, bh * 8, bw * 8)) * (rng.random((3, bh * 8, bw * 8)) < 0.3)
    plan = {"qcoeff": q.astype(np.int32),
            "lf": rng.integers(-40, 400, (3, bh, bw)).astype(np.int32),
            "cfl_x": rng.integers(-20, 20, ((bh + 7) // 8, (bw + 7) // 8)).astype(np.int8),
            "cfl_b": rng.integers(-20, 20, ((bh + 7) // 8, (bw + 7) // 8)).astype(np.int8),
            "lf_factors": (131, 120)}
    hf = rng.integers(1, 4, bmap.shape).astype(np.uint32)
    sh = rng.integers(0, 8, bmap.shape).astype(np.uint8)
    layout = jg.Layout(ctx, w, h, bmap, hf, sh)
    p = jg.Plan(plan["qcoeff"], plan["lf"], plan["cfl_x"], plan["cfl_b"], plan["lf_factors"])
    req = jg.EncodeRequest(global_scale=12000, quant_lf=8, epf_iters=1)
    got = jg.PlanRenderer(ctx).render(layout, p, req, out="xyb")
    rc, want = oracle.reconstruct(w, h, bmap, hf, sh, plan, global_scale=12000, quant_lf=8,
                                  epf_iters=1, out_kind=0)
    assert rc == 0
    assert np.array_equal(got.view(np.uint32), want.view(np.uint32))
