"""wl_rows_product, the C entry with all parts in one array, against exact integers."""
import ctypes

import numpy as np
import pytest

import clwilson_b200 as wl

pytestmark = pytest.mark.gpu
PRIMES = [5, 7, 65537, (1 << 31) - 1, 2147483659, (1 << 47) - 115, 140737488355333, (1 << 61) - 1, (1 << 62) - 57]


def _call(engine, p, parts, out, nparts=None):
    ptr = lambda a: a.ctypes.data if a is not None else None
    return wl.load_library().wl_rows_product(engine._ctx, len(p), ptr(p), len(parts) if nparts is None else nparts,
                                             ptr(parts), ptr(out))


@pytest.mark.parametrize("nparts", [1, 2, 7])
def test_exact(engine, nparts):
    rng = np.random.default_rng(nparts)
    p = np.array(PRIMES * 30, dtype=np.uint64)
    parts = rng.integers(0, 1 << 63, size=(nparts, len(p), 2), dtype=np.uint64) % p[None, :, None]
    out = np.zeros((len(p), 2), dtype=np.uint64)
    assert _call(engine, p, parts, out) == 0
    for i, q in enumerate(map(int, p)):
        want = 1
        for k in range(nparts):
            want = want * (int(parts[k, i, 0]) + q * int(parts[k, i, 1])) % (q * q)
        assert (int(out[i, 0]), int(out[i, 1])) == (want % q, want // q), (q, i)


def test_refusals(engine):
    p = np.array([7, 11], dtype=np.uint64)
    good = np.array([[[1, 2], [3, 4]]], dtype=np.uint64)
    out = np.full((2, 2), 99, dtype=np.uint64)
    assert _call(engine, p, good, out, nparts=0) == -1
    assert _call(engine, p, np.zeros((0, 2, 2), np.uint64), out, nparts=(1 << 16) + 1) == -1
    assert _call(engine, p, np.array([[[7, 0], [0, 0]]], dtype=np.uint64), out) == -1
    assert _call(engine, np.array([7, 10], dtype=np.uint64), good, out) == -1
    assert wl.load_library().wl_rows_product(engine._ctx, 2, p.ctypes.data, 1, None, out.ctypes.data) == -1
    assert (out == 99).all()
    assert wl.load_library().wl_rows_product(engine._ctx, 0, None, 1, None, None) == 0
