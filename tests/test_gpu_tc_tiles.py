"""The tensor-core transforms where their tiling changes: a tile holds 16, 8
or 4 blocks of 8, 16 or 32, and the render takes a CTA per channel as long as
each has an SM; one block, full and partial tiles, both sides of that line,
and frames that cut the last blocks off.  Pixels against the FP32 form (the
reference's): both carry FP32-level error, so they agree to the split form's
bound of 1e-5 for linear pixels."""
import numpy as np
import pytest

import jpxl_gb300 as jg
from jpxl_gb300 import synth

pytestmark = pytest.mark.gpu

CASES = [(8, 1, 1), (8, 17, 1), (8, 30, 27), (8, 40, 31), (16, 1, 1), (16, 9, 1), (16, 21, 20),
         (32, 1, 1), (32, 5, 1), (32, 15, 15)]


@pytest.mark.parametrize("n,cols,rows", CASES)
def test_pixels(ctx, n, cols, rows):
    w, h = cols * n - 3, rows * n - 1
    m = synth.fixed_dct8_map(cols * n, rows * n)
    if n > 8:
        for by in range(rows):
            for bx in range(cols):
                synth.place(m, bx * n // 8, by * n // 8, synth.DCT16 if n == 16 else synth.DCT32)
    rgb = np.random.default_rng(n + cols).integers(0, 256, (h, w, 3)).astype(np.uint8)
    layout = jg.Layout(ctx, w, h, m, 1, 7)
    out = {}
    plan = ctx.encode_transform(layout, rgb, jg.EncodeRequest(global_scale=30000))
    for precision in ("fp32", "bf16x6"):
        req = jg.EncodeRequest(global_scale=30000, precision=precision)
        out[precision] = jg.PlanRenderer(ctx).render(layout, plan, req, out="linear")
        mine = ctx.encode_transform(layout, rgb, req)
        # a coefficient at a decision boundary may fall to the neighbour
        assert np.abs(mine.qcoeff.astype(np.int64) - plan.qcoeff).max() <= 1
        assert (mine.qcoeff != plan.qcoeff).mean() < 1e-3
    assert np.abs(out["bf16x6"] - out["fp32"]).max() < 1e-5
