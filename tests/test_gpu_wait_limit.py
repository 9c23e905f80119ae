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
