"""The error word of a candidate call comes back with its ids: reported once, on both sides of
the limit for results by way of pinned memory, and the calls around it answer."""
import numpy as np
import pytest

import ordvec_b200 as ob
from ordvec_b200._lib import OrdvecError, check, lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nq,m", [(1, 1), (3, 700), (16, 2048), (16, 2049), (40, 3000)])
def test_candidates_report_the_error_word_once(nq, m):
    n, dim = 120_000, 128
    rng = np.random.default_rng(nq)
    sb = ob.SignBitmap(dim)
    sb.add(rng.standard_normal((n, dim)).astype(np.float32))
    q = rng.standard_normal((nq, dim)).astype(np.float32)
    want = sb.top_m_candidates_batched(q, m)
    check(lib().ovb_selftest_arm_tc_error())
    with pytest.raises(OrdvecError) as e:
        sb.top_m_candidates_batched(q, m)
    assert e.value.status == 13 and "timed out" in e.value.message
    again = sb.top_m_candidates_batched(q, m)
    assert all(np.array_equal(a, b) for a, b in zip(again, want))
    for x, row in zip(q[:3], want):
        ham = dim - sb.score_all(x).astype(np.int64)
        assert np.array_equal(row, np.lexsort((np.arange(n), ham))[:m])
