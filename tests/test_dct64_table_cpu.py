"""The 64-point inverse sums its products level by level, which gives the dot
product's terms only if the f32 matrix is symmetric to the bit at every level:
row u's entries over the first 64 >> t columns read the same backwards, or the
same with the other sign, as u >> t is even or odd (t the power of two in u;
level 5 is the last pair)."""
import ctypes as C

import numpy as np

from jpxl_gb300 import _lib, build


def matrix():
    build.build()
    lib = _lib.load()
    m = np.zeros(64 * 64, np.float32)
    assert lib.jpxlg_diag_table(1, m.ctypes.data_as(C.c_void_p)) == m.size
    return m.reshape(64, 64)


def check_symmetric(m):
    for t in range(6):
        n = 64 >> t
        for u in range(0, 64, 1 << t):
            sign = np.float32(-1.0 if (u >> t) & 1 else 1.0)
            assert np.array_equal(m[u, :n], sign * m[u, :n][::-1]), (t, u)


def test_matrix_is_symmetric_at_every_level():
    check_symmetric(matrix())


def test_no_other_table():
    assert _lib.load().jpxlg_diag_table(2, None) == 0
