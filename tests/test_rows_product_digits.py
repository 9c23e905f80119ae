"""What Engine.rows_product hands to the library, part by part (no GPU).

A recording stand-in for the library copies n x 2 64-bit digits from each part's
pointer, as wl_rows_product_parts does.  Parts may be rows with fields of any
integer type, in any byte order or stride, or (n, 2) arrays of any integer type.
"""
import ctypes

import numpy as np
import pytest

import clwilson_b200 as wl

P = [7, 11, 13]
S0, S1 = [1, 2, 3], [4, 5, 6]


class _Recorder:
    def wl_rows_product_parts(self, ctx, n, p, nparts, parts, out):
        self.p = list((ctypes.c_uint64 * n).from_address(p))
        self.parts = [list((ctypes.c_uint64 * (2 * n)).from_address(parts[k])) for k in range(nparts)]
        return 0

    def wl_close(self, ctx):
        pass


def _engine():
    e = wl.Engine.__new__(wl.Engine)
    e._L = _Recorder()
    e._ctx = ctypes.c_void_p()
    return e


def _rows(dtype):
    r = np.zeros(3, dtype=dtype)
    r["p"], r["s0"], r["s1"] = P, S0, S1
    return r


def _field_types():
    yield "rows", wl.ROW_DTYPE
    for t in ("<u4", "<i4", "<i8", ">u8", "<u2", "<f8"):
        yield t, np.dtype([("p", "<u8"), ("s0", t), ("s1", t), ("type", "<u4")])
    yield "mixed", np.dtype([("s1", "<u8"), ("p", "<u4"), ("s0", "<u4"), ("type", "u1")])


@pytest.mark.parametrize("dtype", [d for _, d in _field_types()], ids=[n for n, _ in _field_types()])
@pytest.mark.parametrize("stride", [1, -1, 2])
def test_row_parts(dtype, stride):
    r = _rows(dtype)
    buf = np.zeros(6, dtype=dtype)
    part = buf[::2] if stride == 2 else buf[:3][::stride]
    part[:] = r
    e = _engine()
    e.rows_product([part, _rows(wl.ROW_DTYPE)])
    assert e._L.p == P
    assert e._L.parts == [[1, 4, 2, 5, 3, 6]] * 2


@pytest.mark.parametrize("order", ["C", "F"])
@pytest.mark.parametrize("t", ["<u8", "<u4", "<i8", ">u8", "<f8"])
def test_digit_parts(t, order):
    e = _engine()
    e.rows_product([np.array([[1, 4], [2, 5], [3, 6]], dtype=t, order=order)], p=P)
    assert e._L.p == P and e._L.parts == [[1, 4, 2, 5, 3, 6]]
