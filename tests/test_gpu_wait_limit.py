"""Waits inside the tensor-core products' kernels that run out.

With a limit of zero no wait is waited for: every CTA gives up before its first
matrix instruction, ends the copies that it has in flight and returns.  The call
reports the error, and the context works as before once the limit is back.
"""
import numpy as np
import pytest

import clwilson_b200 as wl

pytestmark = pytest.mark.gpu
LIMIT = 4 * 10**9
TOP = (1 << 62) - 1


# 2 limbs with tails on the tensor cores, 3 limbs, 4 limbs
@pytest.mark.parametrize("lo,hi,qcap", [(10**8, 10**8 + 400000, 0), (10**13, 10**13 + 30000, 1 << 20),
                                        (TOP - 30000, TOP, 1 << 20)])
def test_engine_reports_and_recovers(lo, hi, qcap):
    with wl.Engine(0) as e:
        want, st = e.rows(lo, hi, q_cap=qcap)
        assert st.tensor_macs > 0
        e.set_wait_limit(0)
        for _ in range(2):
            with pytest.raises(wl.WilsonError) as err:
                e.rows(lo, hi, q_cap=qcap)
            assert err.value.code == -2
        e.set_wait_limit(LIMIT)
        got, st = e.rows(lo, hi, q_cap=qcap)
        assert st.tensor_macs > 0 and np.array_equal(got, want)


def _same_as_engine(srv, rid, rows):
    info = srv.wait(rid, 600_000)
    assert info.state == "done", info
    got = srv.rows(rid)
    for f in ("p", "s0", "s1"):
        assert np.array_equal(got[f], rows[f]), f


def test_session_fails_all_running_requests_and_goes_on(engine):
    # two requests take many steps (chunks of at least 65,536 columns, a small step
    # budget); their first step runs out of its waits, so neither may end as done,
    # although the one with columns past 2^32 ends in steps without matrix products
    runs = [(10**13, 10**13 + 30000, 1 << 22), (10**13, 10**13 + 30000, (1 << 32) + (1 << 24))]
    want, st = engine.rows(*runs[0][:2], q_cap=runs[0][2])
    assert st.tensor_macs > 0
    with wl.Server(0, step_cells=1 << 28) as srv:
        srv.set_wait_limit(0)
        ids = [srv.submit(lo, hi, q) for lo, hi, q in runs]
        for rid in ids:
            info = srv.wait(rid, 600_000)
            assert info.state == "failed" and info.rc == -2, info
        srv.set_wait_limit(LIMIT)
        for _ in range(2):
            _same_as_engine(srv, srv.submit(*runs[0]), want)
        st = srv.stats()
        assert st["failed"] == 2 and st["completed"] == 2


def test_session_never_completes_a_request_after_a_bad_step(engine):
    # the limit is cut while a request with columns past 2^32 runs: its last steps
    # hold no matrix products, and it still must not end as done
    lo, hi, q = 10**13, 10**13 + 30000, (1 << 32) + (1 << 31)
    with wl.Server(0, step_cells=1 << 28) as srv:
        srv.set_wait_limit(0)
        first = srv.submit(lo, hi, 1 << 22)
        second = srv.submit(lo, hi, q)
        srv.wait(first, 600_000)
        srv.set_wait_limit(LIMIT)
        third = srv.submit(lo, hi, 1 << 22)
        info = [srv.wait(i, 600_000) for i in (first, second, third)]
        rows, _ = engine.rows(lo, hi, q_cap=1 << 22)
        assert info[0].state == "failed"
        for i, rid, cap in ((info[1], second, q), (info[2], third, 1 << 22)):
            assert i.state in ("failed", "done")
            if i.state == "done":
                want = rows if cap == 1 << 22 else engine.rows(lo, hi, q_cap=cap)[0]
                _same_as_engine(srv, rid, want)
        _same_as_engine(srv, srv.submit(lo, hi, 1 << 22), rows)
