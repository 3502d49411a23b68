"""The encoder at the sizes where its tiling changes, bit for bit against the
restatement: inverse Gaborish tiles of 32, 48 and 64 rows (8, 24 and 40 of
outputs, 104 across) up to the largest frame that gives each an SM of its own
and tiles of 128 beyond it, their edges and remainders, frames of one row or
column; chroma-from-luma CTAs of 512 threads up to a tile per SM and of 256
beyond."""
import numpy as np
import pytest

import jpxl_gb300 as jg
from jpxl_gb300 import synth

pytestmark = pytest.mark.gpu

SIZES = [(1, 90), (90, 1), (2, 41), (3, 200), (200, 3), (103, 39), (104, 40), (105, 41), (107, 80),
         (116, 52), (128, 64), (129, 65), (211, 121), (208, 200), (209, 201), (312, 384),
         (313, 385), (520, 400), (521, 401), (832, 1000)]


@pytest.mark.parametrize("w,h", SIZES)
def test_encode(ctx, oracle, w, h):
    rng = np.random.default_rng(w * 1009 + h)
    rgb = rng.integers(0, 256, (h, w, 3)).astype(np.uint8)
    bmap = synth.mixed_cover(w, h, seed=w + h, rectangles=False)
    hf = rng.integers(1, 9, bmap.shape).astype(np.uint32)
    layout = jg.Layout(ctx, w, h, bmap, hf, 7)
    plan = ctx.encode_transform(layout, rgb, jg.EncodeRequest(global_scale=20000, gaborish=True))
    rc, ref = oracle.encode(rgb, bmap, hf, global_scale=20000, gaborish=True)
    assert rc == 0
    for k in ("qcoeff", "lf", "cfl_x", "cfl_b"):
        assert np.array_equal(getattr(plan, k), ref[k]), k
    assert tuple(plan.lf_factors) == tuple(ref["lf_factors"])
