"""Exact RankQuant batches on both sides of the rule between the sampled filter and the key
matrix (kp = n / 160, 256 queries, 131,072 rows), directly and as a captured plan of a mixed
batch: ids and score bits of the scan that scores every document exactly."""
import numpy as np
import pytest

import ordvec_b200 as ob

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,nq,k", [(40_000, 64, 125), (40_000, 64, 126), (40_000, 256, 300), (40_000, 257, 300),
                                    (131_072, 70, 500), (131_073, 70, 500)])
@pytest.mark.parametrize("bits", [1, 4])
def test_both_sides(monkeypatch, bits, n, nq, k):
    dim = 128
    rng = np.random.default_rng(n + nq + k)
    docs = rng.standard_normal((n, dim)).astype(np.float32)
    docs[100:100 + 3 * k] = docs[5]
    q = (docs[rng.integers(2000, n, nq)] + 0.5 * rng.standard_normal((nq, dim))).astype(np.float32)
    q[1], q[2] = docs[5], 0.0
    rq = ob.RankQuant(dim, bits)
    rq.add(docs)
    monkeypatch.setenv("OVB_RANK_TC", "0")
    monkeypatch.setenv("OVB_ROW_SCORES", "0")
    want = rq.search_asymmetric(q, k)
    monkeypatch.delenv("OVB_RANK_TC")
    monkeypatch.delenv("OVB_ROW_SCORES")
    got = rq.search_asymmetric(q, k)
    assert np.array_equal(got.indices, want.indices)
    assert np.array_equal(got.scores.view(np.uint32), want.scores.view(np.uint32))
    easy = q.copy()
    easy[1] = easy[2] = easy[3]
    monkeypatch.setenv("OVB_RANK_TC", "0")
    monkeypatch.setenv("OVB_ROW_SCORES", "0")
    want = rq.search_asymmetric(easy, k)
    monkeypatch.delenv("OVB_RANK_TC")
    monkeypatch.delenv("OVB_ROW_SCORES")
    for _ in range(3):  # the exact pipeline, then what it left: a captured plan, or itself
        got = ob.search_mixed([rq], np.zeros(nq, np.uint32), np.full(nq, k, np.uint32), easy)
        assert np.array_equal(got.indices, want.indices)
