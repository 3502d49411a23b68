"""The quantizer's nearest-reconstruction choice and the cover search built
on it, bit for bit against the restatement: quantizers from so coarse that
every coefficient falls under the zero threshold to so fine that quotients
leave the table of levels (1024 and beyond) and then the working range, where
both refuse, on noise, whose coefficients
spread over all of them; frames of one block, of partial 32x32 regions and
of odd sizes."""
import numpy as np
import pytest

import jpxl_gb300 as jg
from jpxl_gb300 import synth

pytestmark = pytest.mark.gpu

SCALES = [300, 4000, 60000, 900000, 9000000]


def _noise(w, h, seed):
    return np.random.default_rng(seed).integers(0, 256, (h, w, 3)).astype(np.uint8)


@pytest.mark.parametrize("gs", SCALES)
def test_plan_over_the_quantizer_range(ctx, oracle, gs):
    w, h = 104, 96
    rgb = _noise(w, h, gs % 1009)
    bmap = synth.mixed_cover(w, h, seed=gs, rectangles=False)
    hf = np.random.default_rng(gs).integers(1, 300, bmap.shape).astype(np.uint32)
    req = jg.EncodeRequest(global_scale=gs, gaborish=True)
    layout = jg.Layout(ctx, w, h, bmap, hf, 7)
    rc, ref = oracle.encode(rgb, bmap, hf, global_scale=gs, gaborish=True)
    if rc:  # a target outside the working range: both refuse
        with pytest.raises(jg.JpxlError):
            ctx.encode_transform(layout, rgb, req)
        return
    plan = ctx.encode_transform(layout, rgb, req)
    for k in ("qcoeff", "lf", "cfl_x", "cfl_b"):
        assert np.array_equal(getattr(plan, k), ref[k]), k
    assert tuple(plan.lf_factors) == tuple(ref["lf_factors"])


@pytest.mark.parametrize("w,h", [(1, 1), (8, 8), (9, 7), (31, 33), (32, 32), (40, 24), (65, 47),
                                 (97, 130)])
@pytest.mark.parametrize("gs", SCALES)
def test_cover_of_partial_regions(ctx, oracle, w, h, gs):
    rgb = synth.synthetic_rgb(w, h, seed=w * 3 + h) if min(w, h) > 8 else _noise(w, h, w + h)
    req = jg.EncodeRequest(global_scale=gs, gaborish=True)
    rc, want, _ = oracle.select_blocks(rgb, global_scale=gs, gaborish=True)
    if rc:
        with pytest.raises(jg.JpxlError):
            jg.select_blocks(ctx, rgb, req)
        return
    assert np.array_equal(jg.select_blocks(ctx, rgb, req), want)
