"""The cube roots' and the output levels' short forms give the rule's bits for
every float there is: finite ones of either sign, infinities and NaNs."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu

ALL = 1 << 32
CBRT = {"codec": 0, "metric": 1}
LEVELS = 100


def _wrong(ctx, what, first=0, count=ALL):
    n = C.c_uint64(1)
    ctx.check(ctx.lib.jpxlg_diag_sweep(ctx.handle, what, first, count, C.byref(n)))
    return n.value


@pytest.mark.parametrize("which", list(CBRT))
def test_cube_root_of_every_float(ctx, which):
    assert _wrong(ctx, CBRT[which]) == 0


@pytest.mark.parametrize("bits", [1, 8, 9, 12, 16])
def test_level_of_every_float(ctx, bits):
    assert _wrong(ctx, LEVELS + bits) == 0


def test_bad_sweeps_are_argument_errors(ctx):
    n = C.c_uint64()
    sweep = ctx.lib.jpxlg_diag_sweep
    assert sweep(ctx.handle, LEVELS + 17, 0, 1, C.byref(n)) == -1
    assert sweep(ctx.handle, 2, 0, 1, C.byref(n)) == -1
    assert sweep(ctx.handle, 0, 1, ALL, C.byref(n)) == -1
    assert sweep(ctx.handle, 0, 0, 1, None) == -1
