"""Column products on the tensor cores (wl_tensor.cu), bit for bit against the oracle.

Ranges large enough that every class takes that path, which the call's stats
show (no dense sweep ran although every capped column here is in its regime),
at the edges of the limb widths (p just below 2^31, 2^47 and 2^62), with few
and many rows per 256-column tile, with 5- to 9-bit exponent digits, with
columns cut off at odd places and starting past 2 with a running product.
"""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu
TOP = (1 << 62) - 1


@pytest.fixture(scope="module", autouse=True)
def built():
    oracle.build()


def _same(got, want, sel, fields=("p", "s0", "s1")):
    for f in fields:
        assert np.array_equal(got[f][sel].astype(np.uint64), want[f][sel].astype(np.uint64)), f


@pytest.mark.parametrize("lo,hi,qcap,nsample", [
    ((1 << 31) - 800001, (1 << 31) - 1, (1 << 16) + 1, 200),  # 2 limbs, n up to 2^62, short lists
    ((1 << 47) - 60001, (1 << 47) - 1, (1 << 20) + 7, 6),     # 3 limbs, n up to 2^94
    (10**13, 10**13 + 800000, 1 << 16, 200),                  # 27,000 rows, 5-bit digits
    (10**13, 10**13 + 30000, (1 << 22) - 1, 6),
    (TOP - 8000, TOP, 1 << 24, 6),                            # 46 to 93 rows per class, 9-bit digits
    (TOP - 60000, TOP, 1 << 20, 6),                           # 4 limbs, n up to 2^124
], ids=["2^31", "2^47", "mid-16", "mid-22", "top-few-rows", "top"])
def test_capped_products(engine, lo, hi, qcap, nsample):
    rows, st = engine.rows(lo, hi, q_cap=qcap)
    assert st.dense_column_cells == 0
    sel = (np.linspace(0, len(rows) - 1, nsample).astype(np.uint32) if nsample
           else np.arange(len(rows), dtype=np.uint32))
    want, _ = oracle.search(lo, hi, qcap, rows=sel)
    _same(rows, want, sel)


# the last two have tails of 10^8 integers and more, whose groups run on the
# tensor cores too: at 2 limbs, and with integers on both sides of 2^31
@pytest.mark.parametrize("lo,hi,nsample", [(3 * 10**6, 3 * 10**6 + 60000, 0), (3 * 10**8, 3 * 10**8 + 50000, 12),
                                           (10**8, 10**8 + 400000, 16), (2**32 - 10**5, 2**32 + 150000, 6)])
def test_full_search(engine, lo, hi, nsample):
    rows, st = engine.rows(lo, hi)
    assert (rows["status"] == 0).all() and (rows["rem"] == 0).all()
    sel = np.linspace(0, len(rows) - 1, nsample).astype(np.uint32) if nsample else np.arange(len(rows), dtype=np.uint32)
    want, _ = oracle.search(lo, hi, rows=sel)
    _same(rows, want, sel, ("p", "s0", "s1", "rem", "quot"))


@pytest.mark.parametrize("lo,hi", [(2**33 + 2 * 10**8, 2**33 + 2 * 10**8 + 120000)])
def test_long_tail_equals_short_one(engine, lo, hi):
    # integers past 2^32 in the tail.  T_p! does not depend on where its range
    # starts: the last primes alone have a short tail, which runs cell by cell
    rows, _ = engine.rows(lo, hi)
    last, st = engine.rows(hi - 3000, hi)
    assert (rows["status"] == 0).all() and st.tail_steps < 10**8
    _same(rows[-len(last):], last, np.arange(len(last)), ("p", "s0", "s1", "rem", "quot"))


def test_resumed_products(engine):
    lo, hi, cuts = TOP - 40000, TOP - 1, (1000, 1 << 19, (1 << 21) + 12345)
    part = None
    q = 2
    for c in cuts:
        part, _ = engine.rows_from(lo, hi, q, c, init=part)
        q = c
    whole, st = engine.rows(lo, hi, q_cap=cuts[-1])
    assert st.dense_column_cells == 0
    _same(part, whole, np.arange(len(whole)))
    sel = np.linspace(0, len(whole) - 1, 4).astype(np.uint32)
    want, _ = oracle.search(lo, hi, cuts[-1], rows=sel)
    _same(whole, want, sel)


def test_batch_equals_single_ranges(engine):
    ranges = [(10**9, 10**9 + 30000), (10**12, 10**12 + 9000), (TOP - 20000, TOP), (10**9 + 50, 10**9 + 90)]
    per, _, st = engine.batch(ranges, q_cap=1 << 21)
    assert st.graph_nodes > 0
    for (a, b), r in zip(ranges, per):
        one = engine.search(a, b, q_cap=1 << 21)
        assert r["checksum"] == one.checksum and r["tested"] == one.stats.tested


def test_pieces_of_one_bucket(engine):
    # The class of T = p/2 has 1.7e7 columns, planned at two list entries each and so
    # cut in two pieces; exponents are below 256 from q = 1.6e8 on, so that the pieces
    # together hold fewer entries than one chunk takes.  They share their rows.
    lo, hi, qcap = 8 * 10**10, 8 * 10**10 + 20000, 320 * 10**6
    rows, st = engine.rows(lo, hi, q_cap=qcap)
    assert st.dense_column_cells == 0 and st.tensor_macs > 0
    t = [int(i) for i in range(3) if st.targets[i] > lo // 3]
    hit = np.nonzero(rows["type"] == t[0])[0] if t else np.arange(len(rows))
    sel = hit[np.linspace(0, len(hit) - 1, 8).astype(int)].astype(np.uint32)
    want, _ = oracle.search(lo, hi, qcap, rows=sel)
    _same(rows, want, sel)
