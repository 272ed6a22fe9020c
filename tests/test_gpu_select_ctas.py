"""The whole-GPU select on fewer CTAs than the chip has SMs, as on a partition of it:
slices longer than their stage, one CTA a row, and more rows than CTAs, which take the
other forms.  Ids equal a stable sort's."""
import numpy as np
import pytest

import ordvec_b200 as ob

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ctas", [0, 1, 7, 16, 31])
@pytest.mark.parametrize("nq", [1, 16])
def test_fewer_ctas(monkeypatch, ctas, nq):
    n, dim, m = 120_001, 64, 500
    rng = np.random.default_rng(ctas)
    docs = rng.standard_normal((n, dim)).astype(np.float32)
    queries = rng.standard_normal((nq, dim)).astype(np.float32)
    sb = ob.SignBitmap(dim)
    sb.add(docs)
    monkeypatch.setenv("OVB_BITMAP_TC", "0")
    monkeypatch.setenv("OVB_SELECT_CTAS", str(ctas))
    got = np.stack(sb.top_m_candidates_batched(queries, m))
    for row, q in zip(got, queries):
        ham = dim - sb.score_all(q).astype(np.int64)
        assert np.array_equal(row, np.lexsort((np.arange(n), ham))[:m])
