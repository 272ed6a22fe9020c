"""The per-row select where its last steps change: k at and around powers of two (what lies up
to the last bin fits the final sort, or not), few and many equal keys at the cut, rows of both
block sizes, and k close to the row's length.  Ids equal a stable sort's; the unordered set
of a two-stage search equals the ordered one."""
import numpy as np
import pytest

import ordvec_b200 as ob

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dim", [(3000, 64), (3000, 512), (16_384, 64), (16_385, 256), (40_001, 128)])
def test_select(monkeypatch, n, dim):
    rng = np.random.default_rng(n + dim)
    docs = rng.standard_normal((n, dim)).astype(np.float32)
    docs[n // 2:n // 2 + n // 4] = docs[1]  # a quarter of the row has one key
    q = rng.standard_normal((40, dim)).astype(np.float32)
    q[3] = docs[1]
    sb = ob.SignBitmap(dim)
    sb.add(docs)
    monkeypatch.setenv("OVB_BITMAP_TC", "0")
    order = [np.lexsort((np.arange(n), dim - sb.score_all(x).astype(np.int64))) for x in q]
    for k in (1, 31, 32, 33, 255, 257, 300, 2000, 2048, 2900, 4096, 4097):
        if k > n:
            continue
        got = sb.top_m_candidates_batched(q, k)
        for g, want in zip(got, order):
            assert np.array_equal(g, want[:k]), k


@pytest.mark.parametrize("m", [100, 1000, 2500])
def test_unordered_set(monkeypatch, m):
    n, dim = 20_000, 128
    rng = np.random.default_rng(m)
    docs = rng.standard_normal((n, dim)).astype(np.float32)
    docs[500:900] = docs[7]
    q = (docs[rng.integers(0, n, 40)] + 0.5 * rng.standard_normal((40, dim))).astype(np.float32)
    q[5] = docs[7]
    sb, rq = ob.SignBitmap(dim), ob.RankQuant(dim, 2)
    sb.add(docs)
    rq.add(docs)
    monkeypatch.setenv("OVB_BITMAP_TC", "0")
    cand = sb.top_m_candidates_batched(q, m)
    got = ob.two_stage_search(rq, sb, q, m, 50)
    for i, c in enumerate(cand):
        _, want = rq.search_asymmetric_subset(q[i], np.sort(c).astype(np.uint32), 50)
        assert np.array_equal(got.indices_for_query(i), want)


@pytest.mark.parametrize("n", [39_999, 40_000, 98_303, 98_304])
@pytest.mark.parametrize("nq", [1, 8, 9])
def test_both_sides_of_the_whole_gpu_rule(monkeypatch, n, nq):
    """Ordered integer keys, and unordered ones before a rerank; k whose sort is doubled, and not."""
    dim = 64
    rng = np.random.default_rng(n + nq)
    docs = rng.standard_normal((n, dim)).astype(np.float32)
    q = rng.standard_normal((nq, dim)).astype(np.float32)
    sb, rq = ob.SignBitmap(dim), ob.RankQuant(dim, 1)
    sb.add(docs)
    rq.add(docs)
    monkeypatch.setenv("OVB_BITMAP_TC", "0")
    order = [np.lexsort((np.arange(n), dim - sb.score_all(x).astype(np.int64))) for x in q]
    for k in (100, 800, 1024, 2000, 2048, 4096):
        for g, want in zip(sb.top_m_candidates_batched(q, k), order):
            assert np.array_equal(g, want[:k]), k
    got = ob.two_stage_search(rq, sb, q, 1000, 20)
    for i in range(nq):
        _, want = rq.search_asymmetric_subset(q[i], np.sort(order[i][:1000]).astype(np.uint32), 20)
        assert np.array_equal(got.indices_for_query(i), want)
