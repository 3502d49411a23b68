"""The metric's scratch keeps two counts on the device from kernel to kernel.
Calls that overlap on one scratch (which the interface forbids) spoil their
own scores; what they leave in the counts must not reach a later call."""
import numpy as np
import pytest

import jpxl_gb300 as jg
from jpxl_gb300 import synth

pytestmark = pytest.mark.gpu


def _scales(w, h):
    """reference.rs:90: halved while at least 8 x 8, six levels at most."""
    n = 1
    while n < 6 and min(w, h) >= 8:
        w, h, n = (w + 1) // 2, (h + 1) // 2, n + 1
    return n


@pytest.mark.parametrize("w,h", [(64, 64), (333, 217)])
def test_scores_do_not_depend_on_counts_left_behind(ctx, w, h):
    torch = pytest.importorskip("torch")
    lin = jg.srgb_to_linear_planes(synth.synthetic_rgb(w, h, seed=w))
    noise = np.random.default_rng(w).normal(0.0, 0.03, lin.shape)
    cand = np.ascontiguousarray(np.clip(lin + noise, 0.0, 1.0), dtype=np.float32)
    ref = jg.PrecomputedReference(ctx, lin)
    metric = jg.Ssimulacra2(ctx)
    want = metric.score(ref, cand)
    n = 18 * _scales(w, h)
    cand_dev = torch.from_numpy(cand).cuda()
    out = torch.empty(110, dtype=torch.float64, device="cuda")
    for _ in range(2):
        ctx.check(ctx.lib.jpxlg_diag_scan_words(ctx.handle))
        got = metric.score(ref, cand)
        assert got.score == want.score and got.raw_error == want.raw_error
        assert np.array_equal(got.terms, want.terms)
        out.fill_(float("nan"))
        torch.cuda.synchronize()
        ctx.check(ctx.lib.jpxlg_diag_scan_words(ctx.handle))
        metric.score_static_device(ref, cand_dev.data_ptr(), out.data_ptr())
        ctx.synchronize()
        got = out.cpu().numpy()
        assert got[0] == want.score and got[1] == want.raw_error
        assert np.array_equal(got[2:2 + n], want.terms[:n])
    ref.close()
