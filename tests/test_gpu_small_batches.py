"""Few candidate rows: the rerank form with four lanes a row gives the bits of the
lane-per-row form, for every code width, rows that end inside a lane group, ragged
rows by offsets, and both sides of the dispatch's limit of 8,192 rows."""
import numpy as np
import pytest

import ordvec_b200 as ob

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits,dim", [(1, 128), (1, 1024), (2, 64), (2, 768), (4, 32), (4, 1024)])
def test_rerank_forms_agree_bit_for_bit(bits, dim):
    n = 3000
    docs = ob.synth_docs(bits + dim, n, dim)
    queries, _ = ob.synth_queries(bits + dim, n, 12, dim)
    queries[3] = 0.0
    rq = ob.RankQuant(dim, bits)
    rq.add(docs)
    rng = np.random.default_rng(dim)
    # 12 x 1,000 rows are past the limit: one lane a row
    rows = [rng.permutation(n)[:1000].astype(np.uint32) for _ in range(12)]
    off = np.arange(13, dtype=np.uint64) * 1000
    many = rq.search_asymmetric_subset_batched_serial(queries, off, np.concatenate(rows), 1000)
    for qi, cand in enumerate(rows):  # one query's rows: four lanes a row
        s, i = rq.search_asymmetric_subset(queries[qi], cand, 1000)
        assert np.array_equal(i, many.indices_for_query(qi))
        assert np.array_equal(s.view(np.uint32), many.scores_for_query(qi).view(np.uint32))
    # ragged rows, an empty one among them
    cut = [7, 0, 33, 129, 1]
    off = np.concatenate([[0], np.cumsum(cut)]).astype(np.uint64)
    got = rq.search_asymmetric_subset_batched_serial(queries[:5], off, np.concatenate([r[:c] for r, c in zip(rows, cut)]), 40)
    for qi, c in enumerate(cut):
        k = min(40, c)
        if k:
            s, i = rq.search_asymmetric_subset(queries[qi], rows[qi][:c], 40)
            assert np.array_equal(i, got.indices_for_query(qi)[:k])
            assert np.array_equal(s.view(np.uint32), got.scores_for_query(qi)[:k].view(np.uint32))
        assert np.all(got.indices_for_query(qi)[k:] == -1)


@pytest.mark.parametrize("dim", [4, 100, 1024])
def test_fastscan_tables_of_unusual_queries(orc, dim):
    """Zero, constant, negative-zero and single-spike queries: the table's extremes
    come from whole pairs; scores equal the oracle's bits."""
    n = 500
    docs = np.random.default_rng(dim).standard_normal((n, dim)).astype(np.float32)
    qs = np.zeros((5, dim), np.float32)
    qs[1] = -0.0
    qs[2] = 1.0
    qs[3, dim // 2] = -3.0
    qs[4] = docs[7]
    fs = ob.RankQuantFastscan(dim)
    fs.add(docs)
    got = fs.search(qs, 50)
    ws, wi = orc.fastscan_search(orc.fastscan_pack(docs, dim), n, dim, qs, 50)
    assert np.array_equal(got.indices.reshape(5, -1), wi)
    assert np.array_equal(got.scores.reshape(5, -1).view(np.uint32), np.asarray(ws, np.float32).reshape(5, -1).view(np.uint32))


def test_results_around_the_pinned_limit(orc):
    """10,922 results are the most that come back in pinned memory: one more and one
    less give the same prefix, and the oracle's order."""
    n, dim = 11_000, 64
    docs = ob.synth_docs(3, n, dim)
    q, _ = ob.synth_queries(3, n, 1, dim)
    rq = ob.RankQuant(dim, 2)
    rq.add(docs)
    bm = ob.Bitmap(dim, 16)
    bm.add(docs)
    words = orc.bitmap_encode(docs, dim, 16)
    for ix in (rq, bm):
        search = rq.search_asymmetric if ix is rq else bm.search
        a, b = search(q, 10_922), search(q, 10_923)
        assert np.array_equal(a.indices, b.indices[:10_922])
        assert np.array_equal(a.scores.view(np.uint32), b.scores[:10_922].view(np.uint32))
    ws, wi = orc.bitmap_search(words, n, dim, 16, q, 10_922)
    assert np.array_equal(bm.search(q, 10_922).indices, np.asarray(wi).reshape(-1))
