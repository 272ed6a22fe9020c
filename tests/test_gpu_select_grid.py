"""The whole-GPU select at the edges of its range: the shortest rows it takes, rows
past what the CTAs' shared memory stages, one and several rows per launch, and key
distributions that need no digit, the key digits, and the id digits (all keys equal:
the k lowest positions win).  SignBitmap keys are integers, so ids must equal a
stable sort's, and the cluster form's."""
import numpy as np
import pytest

import ordvec_b200 as ob

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dim,nq,m,spread", [
    (32_768, 64, 1, 1, "random"),
    (32_769, 64, 16, 2048, "random"),     # 16 rows of 9 CTAs
    (40_000, 64, 3, 700, "equal"),        # every key the same
    (150_001, 128, 2, 1000, "two"),       # two values: one above, one below the cut
    (1_200_003, 64, 1, 4096, "random"),   # the most a row may keep
    (7_000_001, 64, 1, 50, "random"),     # a slice longer than its stage
])
def test_select_matches_stable_sort(monkeypatch, n, dim, nq, m, spread):
    rng = np.random.default_rng(n)
    base = rng.standard_normal((min(n, 4096), dim)).astype(np.float32)
    if spread == "equal":
        base[:] = base[0]
    elif spread == "two":
        base[:] = np.where((np.arange(len(base)) % 7 == 0)[:, None], base[0], base[1])
    docs = base[rng.integers(0, len(base), n)] if spread == "random" else base[np.arange(n) % len(base)]
    queries = rng.standard_normal((nq, dim)).astype(np.float32)
    sb = ob.SignBitmap(dim)
    sb.add(docs)
    monkeypatch.setenv("OVB_BITMAP_TC", "0")
    got = np.stack(sb.top_m_candidates_batched(queries, m))
    for row, q in zip(got, queries):
        ham = dim - sb.score_all(q).astype(np.int64)
        assert np.array_equal(row, np.lexsort((np.arange(n), ham))[:m])
    monkeypatch.setenv("OVB_SELECT_WIDE", "0")
    assert np.array_equal(got, np.stack(sb.top_m_candidates_batched(queries, m)))
