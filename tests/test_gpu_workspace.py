"""Device memory that the tensor-core products hold.

Calls with many rows in one class, or many small buckets at once, keep within the
workspace that their planner shares out: constants, group products and lane
products each a slab of rows or a chunk of buckets at a time.
"""
import numpy as np
import pytest
import torch

import clwilson_b200 as wl
import oracle

pytestmark = pytest.mark.gpu
GB = 10**9


def _held(e, call):
    """Device memory that a call on engine e leaves allocated, and its result."""
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    r = call()
    torch.cuda.synchronize()
    return before - torch.cuda.mem_get_info()[0], r


def test_tails_of_many_rows():
    # 292,000 rows in the largest class: 9,100 row tiles, 1.2 GB of constants at once.
    # Every row proves itself (its (p-1)! + 1 is a multiple of p); the oracle checks
    # rows on both sides of the borders of 1,024 row tiles
    lo, hi = 10**6, 11 * 10**6
    oracle.build()
    with wl.Engine(0) as e:
        held, (rows, st) = _held(e, lambda: e.rows(lo, hi))
    assert st.tensor_macs > 0 and st.tail_steps >= 10**8
    assert (rows["status"] == 0).all() and (rows["rem"] == 0).all()
    assert held < 1.2 * GB, held
    sel = []
    for t in range(3):
        idx = np.nonzero(rows["type"] == t)[0]
        for border in range(32768, len(idx), 32768):
            sel += [int(idx[border - 1]), int(idx[border])]
        sel += [int(idx[0]), int(idx[-1])]
    sel = np.array(sorted(sel[::3]), dtype=np.uint32)
    want, _ = oracle.search(lo, hi, rows=sel)
    for f in ("p", "s0", "s1", "rem", "quot"):
        assert np.array_equal(rows[f][sel].astype(np.uint64), want[f][sel].astype(np.uint64)), f


def test_group_products_of_many_buckets():
    # 700 ranges, 2,100 buckets of 3,500 columns: the lane runs of their labels, a label
    # each, pad most of the group tiles (before their bytes counted: 1.17 GB held, 0.82 now)
    lo = (1 << 62) - 10**9
    ranges = [(lo + 10**5 * i, lo + 10**5 * i + 1300) for i in range(700)]
    with wl.Engine(0) as e:
        held, (per, _, st) = _held(e, lambda: e.batch(ranges, q_cap=1 << 15))
        assert st.tensor_macs > 0 and st.dense_column_cells == 0
        assert held < 1.0 * GB, held
        for k in (0, 350, 699):
            one = e.search(*ranges[k], q_cap=1 << 15)
            assert per[k]["checksum"] == one.checksum and per[k]["tested"] == one.stats.tested
