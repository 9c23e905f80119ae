"""Calls on a device with little free memory.

The tensor-core products and the sweeps' split products are planned without asking
for the free memory where they are small.  Where they do not fit after all, the
sweeps run the call, with splits that do.  The rest of the device's memory is held
by one plain allocation; every kernel has run before, so that none is loaded then.
"""
import contextlib
import os

import numpy as np
import pytest
import torch

import clwilson_b200 as wl

pytestmark = pytest.mark.gpu
MB = 1 << 20
TOP = (1 << 62) - 1
CALLS = [(10**7, 10**7 + 150000, 0), (10**13, 10**13 + 200000, 1 << 17), (TOP - 200000, TOP, 1 << 17)]


@contextlib.contextmanager
def free_memory(keep):
    """Leaves about `keep` bytes of the device free."""
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    held = torch.empty(torch.cuda.mem_get_info()[0] - keep, dtype=torch.uint8, device="cuda")
    try:
        yield
    finally:
        del held
        torch.cuda.empty_cache()


def _engine(tensor=True):
    old = os.environ.get("WL_TENSOR")
    os.environ["WL_TENSOR"] = "1" if tensor else "0"
    try:
        return wl.Engine(0)
    finally:
        os.environ.pop("WL_TENSOR")
        if old is not None:
            os.environ["WL_TENSOR"] = old


@pytest.fixture(scope="module")
def expected():
    want = {}
    with _engine() as a, _engine(False) as b:
        for lo, hi, q in CALLS + [(TOP - 200000, TOP, 1 << 20)]:
            want[lo, hi, q], st = a.rows(lo, hi, q_cap=q)
            assert st.tensor_macs > 0
            rows, st = b.rows(lo, hi, q_cap=q)
            assert st.tensor_macs == 0 and np.array_equal(rows, want[lo, hi, q])
    return want


@pytest.mark.parametrize("call", CALLS, ids=["2", "3", "4"])
def test_products_that_do_not_fit(expected, call):
    lo, hi, q = call
    with _engine() as e:
        with free_memory(40 * MB):
            rows, st = e.rows(lo, hi, q_cap=q)
        assert st.tensor_macs == 0 and np.array_equal(rows, expected[call])
        rows, st = e.rows(lo, hi, q_cap=q)
        assert st.tensor_macs > 0 and np.array_equal(rows, expected[call])


def test_split_products_that_do_not_fit(expected):
    lo, hi, q = TOP - 200000, TOP, 1 << 20
    with _engine(False) as e, free_memory(14 * MB):
        rows, _ = e.rows(lo, hi, q_cap=q)
    assert np.array_equal(rows, expected[lo, hi, q])


def test_resumed_and_batched_calls(expected):
    lo, hi, q = CALLS[1]
    with _engine() as e:
        with free_memory(40 * MB):
            part, _ = e.rows_from(lo, hi, 2, 10007)
            rows, st = e.rows_from(lo, hi, 10007, q, init=part)
            assert st.tensor_macs == 0
            _, _, st = e.batch([(lo, hi), (lo + 10**6, lo + 10**6 + 200)], q_cap=q)
            assert st.tensor_macs == 0
    for f in ("p", "s0", "s1"):
        assert np.array_equal(rows[f], expected[CALLS[1]][f])


def test_session(expected):
    with wl.Server(0, pool_bytes=64 * MB) as srv:
        # a first request, with the memory free: the session plans with the products
        small = (10**13, 10**13 + 20000, 1 << 17)
        first = srv.submit(*small)
        assert srv.wait(first, 600_000).state == "done"
        with free_memory(24 * MB):
            ids = [srv.submit(*CALLS[1]), srv.submit(*small)]
            infos = [srv.wait(i, 600_000) for i in ids]
        assert [i.state for i in infos] == ["done", "done"], infos
        for f in ("p", "s0", "s1"):
            assert np.array_equal(srv.rows(ids[0])[f], expected[CALLS[1]][f])
            assert np.array_equal(srv.rows(ids[1])[f], srv.rows(first)[f])
        again = srv.submit(*CALLS[1])
        assert srv.wait(again, 600_000).state == "done"
        assert np.array_equal(srv.rows(again)["s1"], expected[CALLS[1]]["s1"])


def test_column_table_that_does_not_fit():
    # a table for 5e8 takes 110 MB: the call fails, and the smaller table that it was to
    # replace is sieved again by the next call that needs it
    small, large = (10**6, 10**6 + 2000), (10**9, 10**9 + 100)
    with wl.Engine(0) as e:
        want, _ = e.rows(*small)
        with free_memory(30 * MB):
            with pytest.raises(wl.WilsonError) as err:
                e.rows(*large)
            assert err.value.code == -8
            rows, _ = e.rows(*small)
            assert np.array_equal(rows, want)
        rows, _ = e.rows(*large)
        assert (rows["status"] == 0).all() and (rows["rem"] == 0).all()


def test_session_whose_table_does_not_fit(expected):
    # a request that needs the larger table fails; the one that is running, on the sweeps
    # in small steps, goes on with the table that it was admitted with
    lo, hi, q = 10**13, 10**13 + 200000, 1 << 27
    with _engine(False) as e:
        want, _ = e.rows(lo, hi, q_cap=q)
    os.environ["WL_TENSOR"] = "0"
    try:
        srv = wl.Server(0, pool_bytes=64 * MB, step_cells=1 << 26)
    finally:
        os.environ.pop("WL_TENSOR")
    with srv:
        long = srv.submit(lo, hi, q)
        while srv.poll(long).state == "queued":
            pass
        with free_memory(40 * MB):
            large = srv.submit(10**9, 10**9 + 100)
            info = srv.wait(large, 600_000)
            assert info.state == "failed" and info.rc == -8
            assert srv.poll(long).state == "active"
            assert srv.wait(long, 600_000).state == "done"
        got = srv.rows(long)
        for f in ("p", "s0", "s1"):
            assert np.array_equal(got[f], want[f])
        again = srv.submit(10**9, 10**9 + 100)
        assert srv.wait(again, 600_000).state == "done"
