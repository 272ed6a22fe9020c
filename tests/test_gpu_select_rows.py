"""The select of one row per CTA: short and long rows, few and many of a row's entries,
integer keys of few values (ties by id), floats, equal keys, keys an ulp apart beside far
outliers, and repeated candidates.  Exact: ids equal a stable sort's, and a smaller k is
a prefix of the full sort's."""
import numpy as np
import pytest

import ordvec_b200 as ob

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [33, 2047, 16384, 16385, 40_000])
@pytest.mark.parametrize("spread", ["random", "equal", "two"])
def test_integer_keys(monkeypatch, n, spread):
    dim, nq = 64, 40  # too many rows for the forms that share one
    rng = np.random.default_rng(n)
    docs = rng.standard_normal((n, dim)).astype(np.float32)
    if spread == "equal":
        docs[:] = docs[0]
    elif spread == "two":
        docs[:] = np.where((np.arange(n) % 7 == 0)[:, None], docs[0], docs[1])
    queries = rng.standard_normal((nq, dim)).astype(np.float32)
    sb = ob.SignBitmap(dim)
    sb.add(docs)
    monkeypatch.setenv("OVB_BITMAP_TC", "0")
    want = np.stack([np.lexsort((np.arange(n), dim - sb.score_all(q).astype(np.int64))) for q in queries])
    for m in sorted({1, 31, min(n, 300), min(n, 2048), min(n, 2049), min(n, 5000), n - 1, n}):
        if m <= 5000 or n < 20_000:
            assert np.array_equal(np.stack(sb.top_m_candidates_batched(queries, m)), want[:, :m]), m


@pytest.mark.parametrize("kind", ["random", "outliers"])
@pytest.mark.parametrize("rows", [1, 20])
def test_float_keys_and_repeated_candidates(kind, rows):
    dim, n = 128, 3500  # as many documents as candidates a row
    rng = np.random.default_rng(rows)
    docs = rng.standard_normal((n, dim)).astype(np.float32)
    if kind == "outliers":  # scores in a narrow band, and a few documents far away
        docs[:] = docs[0] + 1e-3 * docs
        docs[5], docs[6] = -docs[0], np.abs(docs[0])
    rq = ob.RankQuant(dim, 4)
    rq.add(docs)
    q = docs[rng.integers(0, n, rows)]
    cand = [np.concatenate([rng.integers(0, n, 2500), np.full(700, 11), rng.permutation(n)[:300]]).astype(np.uint32)
            for _ in range(rows)]
    off = np.arange(rows + 1, dtype=np.uint64) * 3500
    full = rq.search_asymmetric_subset_batched_serial(q, off, np.concatenate(cand), 3500)
    for qi in range(rows):
        s, i = full.scores_for_query(qi), full.indices_for_query(qi)
        assert np.array_equal(np.lexsort((i, -s.astype(np.float64))), np.arange(3500))
        assert np.array_equal(np.sort(i), np.sort(cand[qi]))
    for k in (1, 100, 257, 1000, 2048, 3499):
        got = rq.search_asymmetric_subset_batched_serial(q, off, np.concatenate(cand), k)
        for qi in range(rows):
            assert np.array_equal(got.indices_for_query(qi), full.indices_for_query(qi)[:k])
            assert np.array_equal(got.scores_for_query(qi), full.scores_for_query(qi)[:k])
