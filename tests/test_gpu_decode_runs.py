"""Runs of one decode batch in either memory, in any order: a host run after a
device run that nothing waited for, NULL entries, no outputs at all."""
import ctypes as C
from pathlib import Path

import numpy as np
import pytest

import jpxl_gb300 as jg

pytestmark = pytest.mark.gpu

GOLDEN = Path(__file__).resolve().parent / "golden" / "codestream"
NAMES = ["06_gradient_300x200_lossy", "52_vardct_mixed_gray_128x128_filters_d1",
         "63_vardct_outofgamut_rgb_64x64_nofilters_d4", "72_lfframe_gray_128x128_nofilters"]


@pytest.mark.parametrize("precision", ["fp32", "bf16x6"])
@pytest.mark.parametrize("lanes", [1, 3])
def test_device_and_host_runs_alternate(ctx, precision, lanes):
    torch = pytest.importorskip("torch")
    streams = [jg.Codestream((GOLDEN / (n + ".jxl")).read_bytes()) for n in NAMES * 6]
    batch = jg.DecodeBatch(ctx, streams, "srgb8", lanes=lanes, precision=precision)
    run = ctx.lib.jpxlg_decode_batch_run
    want = [b.copy() for b in batch.run()]
    dev = [torch.zeros(w.size, dtype=torch.uint8, device="cuda") for w in want]
    torch.cuda.synchronize()
    ptrs = (C.c_void_p * len(dev))(*[t.data_ptr() for t in dev])
    for rnd in range(3):
        for b in batch.buffers:
            b.fill(7)
        ctx.check(run(ctx.handle, batch.handle, ptrs, jg.MEM_DEVICE))
        some = (C.c_void_p * len(want))(*[None if i % 3 == rnd else b.ctypes.data
                                          for i, b in enumerate(batch.buffers)])
        ctx.check(run(ctx.handle, batch.handle, some, jg.MEM_HOST))
        for i, (b, w) in enumerate(zip(batch.buffers, want)):
            assert np.array_equal(b, np.full_like(w, 7) if i % 3 == rnd else w), (rnd, i)
        for t, w in zip(dev, want):
            assert np.array_equal(t.cpu().numpy(), w.ravel())
            t.zero_()
        ctx.check(run(ctx.handle, batch.handle, None, jg.MEM_HOST))
        torch.cuda.synchronize()
    batch.close()
