"""The blocks only decoded streams have: sides of 64 and the 8x8 special
transforms, each over whole frames and frames that cut the last blocks off,
against the restatement's parts put together here (jpxl-core varblock.rs:817,
reconstruct.rs:27-96, dct.rs:678 and :982), and the kernel that lays a staged
stream out on the device, at the three widths of its coefficients."""
import ctypes as C
import json
from pathlib import Path

import numpy as np
import pytest

import jpxl_gb300 as jg
from jpxl_gb300 import _lib
from test_dct64_table_cpu import check_symmetric, matrix

pytestmark = pytest.mark.gpu

F = np.float32
BIAS = (F(1.0) - F(0.054650073), F(1.0) - F(0.0700545), F(1.0) - F(0.049935103))
AFV = np.array(json.loads((Path(__file__).resolve().parent / "golden" /
                           "reference_constants.json").read_text())["AFV_BASIS"], np.float64)
# DctSelect: block rows, block columns, place of its matrix in a channel's table
LARGE = {18: (8, 8, 2304), 19: (8, 4, 6400), 20: (4, 8, 6400)}
# DctSelect: kind of the special transform, place of its matrix
SPECIAL = {1: (2, 8448), 2: (1, 2240), 3: (3, 8512), 12: (5, 8576), 13: (4, 8576), 14: (6, 8640),
           15: (7, 8640), 16: (8, 8640), 17: (9, 8640)}
SCALE, QUANT_LF = 12000, 8


def _tables():
    t = np.zeros(_lib.load().jpxlg_diag_table(0, None), np.float32)
    _lib.load().jpxlg_diag_table(0, t.ctypes.data)
    return t.reshape(3, -1)


def _frame(sel, brows, bcols, cols, rows, cut, seed):
    """A frame of one kind of block: size, cover and a plan."""
    w, h = cols * bcols * 8 - cut, rows * brows * 8 - (cut * 5) % 8
    bmap = np.full((rows * brows, cols * bcols), sel, np.uint8)
    bmap[::brows, ::bcols] |= jg.ORIGIN
    rng = np.random.default_rng(seed)
    bh, bw = bmap.shape
    q = rng.integers(-6, 7, (3, bh * 8, bw * 8)) * (rng.random((3, bh * 8, bw * 8)) < 0.2)
    tiles = ((bh + 7) // 8, (bw + 7) // 8)
    plan = jg.Plan(q.astype(np.int32), rng.integers(-40, 400, (3, bh, bw)).astype(np.int32),
                   rng.integers(-20, 20, tiles).astype(np.int8),
                   rng.integers(-20, 20, tiles).astype(np.int8), (131, 120))
    hf = rng.integers(1, 4, bmap.shape).astype(np.uint32)
    return w, h, bmap, plan, hf


def _lf(plan):
    """reconstruct.rs:84 and the LF CfL (plan-render lib.rs:1314)."""
    d = [F(65536.0 * float(F(wt) / F(128.0)) / (float(SCALE) * QUANT_LF)) *
         plan.lf[c].astype(np.float32) for c, wt in enumerate((1 / 32, 1 / 4, 1 / 2))]
    kx = F(plan.lf_factors[0] - 128) / F(84.0)
    kb = F(1.0) + F(plan.lf_factors[1] - 128) / F(84.0)
    return [d[0] + kx * d[1], d[1], d[2] + kb * d[1]]


def _coefficients(oracle, plan, hf, table, by, bx, brows, bcols):
    """A block's dequantized landscape coefficients, HF CfL applied."""
    lib = oracle.load()
    mul = F(lib.orc_hf_multiplier(SCALE, int(hf[by, bx])))
    co = []
    for c in range(3):
        q = plan.qcoeff[c, by * 8:(by + brows) * 8, bx * 8:(bx + bcols) * 8]
        q = q.T if brows > bcols else q
        lut = np.array([lib.orc_bias_adjust(int(v), float(BIAS[c]), 0.145) for v in range(-8, 9)],
                       np.float32)
        co.append(lut[q + 8] * mul * table[c].reshape(q.shape))
    kx = F(plan.cfl_x[by // 8, bx // 8]) / F(84.0)
    kb = F(1.0) + F(plan.cfl_b[by // 8, bx // 8]) / F(84.0)
    return [co[0] + kx * co[1], co[1], co[2] + kb * co[1]]


def _inverse(lib, m64, n, a):
    """dct.rs:749 down every column of a: n = 64 an f64 dot product rounded
    once (:678), 32 the butterflies."""
    if n == 64:
        acc = np.zeros(a.shape, np.float64)
        for j in range(64):
            acc += m64[j].astype(np.float64)[:, None] * a[j].astype(np.float64)[None, :]
        return acc.astype(np.float32) * F(8.0)
    out = np.empty_like(a)
    for x in range(a.shape[1]):
        col = np.ascontiguousarray(a[:, x])
        lib.orc_idct_1d(C.c_void_p(col.ctypes.data), n)
        out[:, x] = col
    return out


def _render(ctx, w, h, bmap, plan, hf):
    layout = jg.Layout(ctx, w, h, bmap, hf, np.full(bmap.shape, 4, np.uint8))
    req = jg.EncodeRequest(global_scale=SCALE, quant_lf=QUANT_LF)
    return jg.PlanRenderer(ctx).render(layout, plan, req, out="xyb")


@pytest.mark.parametrize("cols,rows,cut", [(1, 1, 0), (3, 2, 0), (2, 2, 3)])
@pytest.mark.parametrize("sel", list(LARGE))
def test_sides_of_64(ctx, oracle, sel, cols, rows, cut):
    """The kernel's sum and the reference's both lie within about 2^-46 of the
    terms' magnitudes of the exact dot product, so one in a few hundred
    thousand of the first pass's sums may round the other way, an ulp, and
    take some of its line's 64 samples with it: at least 99.9 % of the samples
    equal to the bit, none further off than two ulps of the block's largest."""
    brows, bcols, place = LARGE[sel]
    w, h, bmap, plan, hf = _frame(sel, brows, bcols, cols, rows, cut, 100 * sel + cols)
    lib, m64 = oracle.load(), matrix()
    check_symmetric(m64)
    table = _tables()[:, place:place + 64 * brows * bcols]
    lf = _lf(plan)
    cy, cx = min(brows, bcols), max(brows, bcols)
    sf = [np.array([lib.orc_scale_f(i, n) for i in range(n)], np.float32) for n in (cy, cx)]
    want = np.zeros((3, rows * brows * 8, cols * bcols * 8), np.float32)
    got = _render(ctx, w, h, bmap, plan, hf)
    for by in range(0, rows * brows, brows):
        for bx in range(0, cols * bcols, bcols):
            co = _coefficients(oracle, plan, hf, table, by, bx, brows, bcols)
            for c in range(3):
                rect = lf[c][by:by + brows, bx:bx + bcols]
                rect = oracle.dct_2d(rect.T if brows > bcols else rect)
                co[c][:cy, :cx] = rect * sf[0][:, None] * sf[1][None, :]
                s = co[c].T if bcols > brows else co[c]  # bcols x brows blocks
                a = _inverse(lib, m64, bcols * 8, np.ascontiguousarray(s))
                a = _inverse(lib, m64, brows * 8, np.ascontiguousarray(a.T))
                ys, xs = slice(by * 8, (by + brows) * 8), slice(bx * 8, (bx + bcols) * 8)
                want[c, ys, xs] = a
                g, v = got[c, ys, xs], a[:min(h, (by + brows) * 8) - by * 8,
                                         :min(w, (bx + bcols) * 8) - bx * 8]
                assert np.abs(g - v).max() <= 2 * np.spacing(np.abs(v).max())
    want = want[:, :h, :w]
    same = (got.view(np.uint32) == want.view(np.uint32)).mean()
    print(f"DctSelect {sel}, {w}x{h}: {100 * same:.4f} % of the samples the same bits")
    assert same >= 0.999


@pytest.mark.parametrize("cols,rows,cut", [(1, 1, 0), (7, 5, 3)])
@pytest.mark.parametrize("sel", list(SPECIAL))
def test_special_blocks_in_a_frame(ctx, oracle, sel, cols, rows, cut):
    kind, place = SPECIAL[sel]
    w, h, bmap, plan, hf = _frame(sel, 1, 1, cols, rows, cut, 100 * sel + cols)
    table = _tables()[:, place:place + 64]
    lf = _lf(plan)
    sf = F(oracle.load().orc_scale_f(0, 1))
    want = np.zeros((3, rows * 8, cols * 8), np.float32)
    for by in range(rows):
        for bx in range(cols):
            co = _coefficients(oracle, plan, hf, table, by, bx, 1, 1)
            for c in range(3):
                co[c][0, 0] = lf[c][by, bx] * sf * sf
                want[c, by * 8:by * 8 + 8, bx * 8:bx * 8 + 8] = oracle.special_block(kind, co[c],
                                                                                     AFV)
    got = _render(ctx, w, h, bmap, plan, hf)
    assert np.array_equal(got, want[:, :h, :w])


@pytest.mark.parametrize("n,rest", [(64, 0), (64, 16), (64 * 331, 4096 + 16)])
@pytest.mark.parametrize("dtype", [np.int8, np.int16, np.int32])
def test_unstage_widths(ctx, dtype, n, rest):
    info = np.iinfo(dtype)
    rng = np.random.default_rng(n + rest)
    q = rng.integers(info.min, info.max, n, endpoint=True).astype(dtype)
    q[:4] = (info.min, info.max, -1, 1)
    q[-3:] = (info.max, info.min, -2)
    tail = rng.integers(0, 256, rest).astype(np.uint8)
    src = np.concatenate([q.view(np.uint8), tail])
    dst = np.zeros(4 * n + rest, np.uint8)
    ctx.check(ctx.lib.jpxlg_diag_unstage(ctx.handle, q.itemsize, src.ctypes.data, n, rest,
                                         dst.ctypes.data))
    assert np.array_equal(dst[:4 * n].view(np.int32), q.astype(np.int32))
    assert np.array_equal(dst[4 * n:], tail)
