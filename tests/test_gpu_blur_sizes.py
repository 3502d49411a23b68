"""SSIMULACRA2 at the edges of its kernels' tiles, against the restatement.

Widths around the row pass's segments (128 a line, an odd number of samples
each), its groups of four outputs and its 16-byte rows; heights around the
column pass's 64-row segments and 32-row tiles; strips of 32 columns; the
pyramid's 64 x 64 tiles; the widest line.

The restatement sums the metric in f64 and the kernels in double-float, and
their f32 blur outputs differ only where the reference's f64 noise decides a
rounding (3 samples in 10^4, one ulp).  One ulp (2^-24 of a sample near one)
moves a pixel's SSIM term by at most 2^-24 / C2 = 6.6e-5, so the mean over a
frame by 2e-8 and the score, whose derivative in a term stays below 2000
points, by less than 1e-4.
"""
import numpy as np
import pytest

import jpxl_gb300 as jg
from jpxl_gb300 import synth

pytestmark = pytest.mark.gpu

SIZES = [(8, 8), (9, 33), (31, 64), (32, 65), (33, 129), (127, 63), (128, 66), (129, 31),
         (255, 130), (511, 17), (512, 96), (516, 200), (645, 97), (1022, 40), (2051, 72),
         (4097, 34), (8192, 9)]


@pytest.mark.parametrize("w,h", SIZES)
def test_score_at_tile_edges_matches_the_restatement(ctx, oracle, w, h):
    src = jg.srgb_to_linear_planes(synth.synthetic_rgb(w, h, seed=w + h))
    rng = np.random.default_rng(w * 7 + h)
    cand = np.clip(src + rng.normal(0.0, 0.02, src.shape), 0.0, 1.0).astype(np.float32)
    want, _, _ = oracle.ssim2(src, cand)
    ref = jg.PrecomputedReference(ctx, src)
    got = jg.Ssimulacra2(ctx).score(ref, cand).score
    assert abs(got - want) < 1e-4, (got, want)
    # a second pass over the same scratch, and the pair form, agree exactly
    assert jg.Ssimulacra2(ctx).score(ref, cand).score == got
    assert jg.score_pair(ctx, src, cand) == got
    ref.close()
