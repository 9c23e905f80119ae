"""The sweeps' kernels, on contexts that run nothing else (WL_TENSOR=0 when opened).

Most calls take the tensor-core products by themselves; the sweeps still run buckets
of few rows or columns, columns past 2^32 and devices short of memory, in the
variants that wl_autotune chooses among.  Every call here checks in its stats that
the sweeps ran, and that they ran the columns in the regime that it is about.
"""
import contextlib
import os

import numpy as np
import pytest

import clwilson_b200 as wl
import oracle

pytestmark = pytest.mark.gpu
TOP = (1 << 62) - 1


@contextlib.contextmanager
def sweeps_alone():
    old = os.environ.get("WL_TENSOR")
    os.environ["WL_TENSOR"] = "0"
    try:
        yield
    finally:
        if old is None:
            del os.environ["WL_TENSOR"]
        else:
            os.environ["WL_TENSOR"] = old


@pytest.fixture(scope="module")
def eng():
    with sweeps_alone():
        e = wl.Engine(0)
    yield e
    e.close()


@pytest.fixture(scope="module")
def big_rows():
    # about 2,200 primes: buckets of more than 512 rows take two and four rows per thread
    oracle.build()
    rows, _ = oracle.search(10**6, 10**6 + 30000)
    return rows


def _same(got, want, fields=("p", "s0", "s1")):
    for f in fields:
        assert np.array_equal(got[f].astype(np.uint64), want[f].astype(np.uint64)), f


def test_route_belongs_to_the_context(eng, engine):
    lo, hi, q = 10**13, 10**13 + 30000, 1 << 20
    a, sa = eng.rows(lo, hi, q_cap=q)
    b, sb = engine.rows(lo, hi, q_cap=q)
    assert sa.tensor_macs == 0 and sa.dense_column_cells > 0
    assert sb.tensor_macs > 0 and sb.dense_column_cells == 0
    assert np.array_equal(a, b)


@pytest.mark.parametrize("kernel", [0, 1, 2, 3, 4, 5, 6])
@pytest.mark.parametrize("hstep", [4, 16])
def test_dense_variants(eng, golden, kernel, hstep):
    eng.tuning = {"dense_kernel": [kernel] * 3, "dense_hstep": [hstep] * 3}
    for lo, hi in [(10**13, 10**13 + 10**7), (TOP - 10**7, TOP)]:
        case = next(c for c in golden["capped"] if c["pmin"] == lo)
        rows, st = eng.rows(lo, hi, q_cap=1 << 16)
        assert st.tensor_macs == 0 and st.dense_column_cells > 0
        byp = {int(p): i for i, p in enumerate(rows["p"])}
        for w in case["rows"]:
            r = rows[byp[w["p"]]]
            assert (int(r["s0"]), int(r["s1"])) == (w["s0"], w["s1"]), w["p"]


@pytest.mark.parametrize("variant", [0, 1, 2, 3])
@pytest.mark.parametrize("rpt", [1, 2, 4])
@pytest.mark.parametrize("merge", [1, 10**6])
def test_sparse_variants_full_search(eng, golden, big_rows, variant, rpt, merge):
    eng.tuning = {"sparse_variant": [variant] * 3, "sparse_rpt": [rpt] * 3, "merge_cta_min": merge,
                  "dense_kernel": [0] * 3, "dense_hstep": [8] * 3}
    rows, st = eng.rows(10**6, 10**6 + 30000)
    assert st.tensor_macs == 0
    _same(rows, big_rows, ("p", "s0", "s1", "rem", "quot"))
    g = golden["range_1e5"]
    res = eng.search(g["pmin"], g["pmax"])
    assert res.lines() == g["lines"] and "%016X" % res.checksum == g["checksum"] and res.stats.tensor_macs == 0


# buckets of 1 to 40 rows: a tile's width is the bucket's own row count up to 32, so
# that the CTA's last threads may belong to no split
@pytest.mark.parametrize("kernel", [0, 2, 4, 5])
@pytest.mark.parametrize("lo,widths,q", [(10**13, range(100, 2500, 170), 1 << 14), (TOP - 10**6, range(150, 3400, 230), 1 << 13),
                                         (10**9, range(80, 1700, 120), 1 << 15)], ids=["3", "4", "2"])
def test_narrow_buckets(eng, kernel, lo, widths, q):
    oracle.build()
    eng.tuning = {"dense_kernel": [kernel] * 3, "dense_hstep": [8] * 3, "sparse_variant": [1] * 3,
                  "sparse_rpt": [2] * 3, "merge_cta_min": 64}
    seen = set()
    for w in widths:
        rows, st = eng.rows(lo, lo + w, q_cap=q)
        assert st.tensor_macs == 0 and st.dense_column_cells > 0
        want, _ = oracle.search(lo, lo + w, q)
        _same(rows, want)
        seen |= set(st.per_class)
    assert len([n for n in seen if 8 < n <= 40 and n & (n - 1)]) >= 8


@pytest.mark.parametrize("lo,hi", [(200, 564), (10**6, 10**6 + 900), (10**7, 10**7 + 1000), (2**31 - 700, 2**31 + 700)])
def test_narrow_full_searches(eng, lo, hi):
    oracle.build()
    eng.tuning = {"dense_kernel": [4] * 3, "sparse_variant": [1] * 3, "sparse_rpt": [2] * 3, "merge_cta_min": 64}
    rows, st = eng.rows(lo, hi)
    assert st.tensor_macs == 0
    sel = np.linspace(0, len(rows) - 1, min(len(rows), 24)).astype(np.uint32)
    want, _ = oracle.search(lo, hi, rows=sel)
    _same(rows[sel], want[sel], ("p", "s0", "s1", "rem", "quot"))


def test_call_with_both_routes(eng, engine):
    # about 880 ranges of one or two rows a class, which the sweeps run (those of 1,000
    # that hold primes), beside one of 10,000 rows
    oracle.build()
    narrow = [(TOP - 10**9 + 10**5 * i, TOP - 10**9 + 10**5 * i + 90) for i in range(1000)]
    ranges = [r for r in narrow if len(oracle.list_primes(*r))] + [(TOP - 430000, TOP)]
    per, _, st = engine.batch(ranges, q_cap=1 << 16)
    assert st.tensor_macs > 0 and st.dense_column_cells > 0
    want, _, st = eng.batch(ranges, q_cap=1 << 16)
    assert st.tensor_macs == 0
    for a, b in zip(per, want):
        assert a == b


def test_session_on_the_sweeps(eng, engine):
    keys = [(10**13, 10**13 + 10000, 1 << 20), (TOP - 20000, TOP, 1 << 20), (10**8, 10**8 + 4000, 0),
            (10**13, 10**13 + 300, 1 << 20)]
    with sweeps_alone():
        srv = wl.Server(0, step_cells=1 << 24)
    with srv:
        ids = [srv.submit(*k) for k in keys]
        for rid, (lo, hi, q) in zip(ids, keys):
            assert srv.wait(rid, 600_000).state == "done"
            want, st = engine.rows(lo, hi, q_cap=q)
            _same(srv.rows(rid), want)


def test_tuning_times_the_sweeps(engine):
    # what autotune reports for a caller's ranges is the sweeps' time, here tens of
    # times that of the call itself
    r, q = (TOP - 50000, TOP), 1 << 24
    with sweeps_alone():
        e = wl.Engine(0)
    with e:
        e.rows(*r, q_cap=q)
        sweeps = min(e.rows(*r, q_cap=q)[1].ms_sweep for _ in range(3))
    with wl.Engine(0) as e:
        e.rows(*r, q_cap=q)
        call = min(e.rows(*r, q_cap=q)[1].ms_sweep for _ in range(3))
        assert call < sweeps / 5
        t = e.autotune([r], q_cap=q)
        assert t["ms"][2] > sweeps / 2
        assert e.rows(*r, q_cap=q)[1].tensor_macs > 0          # the context's own route is back
