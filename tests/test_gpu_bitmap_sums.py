"""The FP4 filter's 16-bit sums at the ends of their range: documents that agree and
disagree with a query in every bit, rows of 255 words (the longest) and of 256 (f32
sums), more kept documents than a warp's list holds, and one to 448 queries.  Candidates
equal the CUDA-core popcount scan's exactly."""
import numpy as np
import pytest

import ordvec_b200 as ob

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind,dim,n,nq,m", [
    ("sign", 64, 3000, 1, 40), ("sign", 16320, 2500, 17, 60), ("sign", 16384, 2500, 17, 60),
    ("bitmap", 16320, 1500, 33, 50), ("bitmap", 16384, 1500, 33, 50),
    ("sign", 512, 6001, 448, 3000),  # half of all documents are kept
])
def test_extreme_sums(monkeypatch, kind, dim, n, nq, m):
    rng = np.random.default_rng(dim + nq)
    docs = rng.standard_normal((n, dim), dtype=np.float32)
    queries = rng.standard_normal((nq, dim), dtype=np.float32)
    for i in range(0, n - 4, n // 50):
        docs[i] = queries[i % nq]         # every bit agrees
        docs[i + 1] = -queries[i % nq]    # none does
        docs[i + 2] = docs[i]             # ties
    ix = ob.Bitmap(dim, dim // 2) if kind == "bitmap" else ob.SignBitmap(dim)
    ix.add(docs)
    monkeypatch.setenv("OVB_FASTSCAN_FILTER", "1")
    monkeypatch.setenv("OVB_BITMAP_TC", "1")
    got = np.stack(ix.top_m_candidates_batched(queries, m))
    monkeypatch.setenv("OVB_BITMAP_TC", "0")
    assert np.array_equal(got, np.stack(ix.top_m_candidates_batched(queries, m)))
