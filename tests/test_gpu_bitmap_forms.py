"""The bitmap-family filter on the FP4 tensor cores over the row lengths and
batch sizes where its forms change: rows of one K-block and less, odd word
counts (8-byte copies), resident rows in two halves, in one, and the ring; rows
beyond 16 words; one and several query tiles; ring depths from 4 to 6 stages; and
a partial last document tile.  Candidates are integers and ids, so they equal
the CUDA-core popcount scan's exactly, ties included."""
import numpy as np
import pytest

import ordvec_b200 as ob

pytestmark = pytest.mark.gpu


def _index(kind, dim, docs):
    ix = {"bitmap": lambda: ob.Bitmap(dim, max(dim // 4, 1)), "sign": lambda: ob.SignBitmap(dim),
          "multibucket": lambda: ob.MultiBucketBitmap(dim, 2)}[kind]()
    ix.add(docs)
    return ix


def _top_m(ix, kind, queries, m):
    if kind == "multibucket":
        return ix.top_m_bilinear_batched(queries, ix.diagonal_weights(), m)
    return np.stack(ix.top_m_candidates_batched(queries, m))


@pytest.mark.parametrize("kind,dim,n,nq", [
    ("bitmap", 64, 40_001, 300),       # one word: a quarter of one K-block, resident, two halves
    ("sign", 192, 40_001, 70),         # three words: 8-byte copies, ring
    ("bitmap", 320, 70_001, 470),      # five words, two K-blocks, three query tiles
    ("sign", 768, 45_000, 225),        # twelve words: resident in two halves, two query tiles
    ("sign", 1024, 45_000, 450),       # sixteen words: resident once
    ("sign", 1024, 33_333, 16),        # ring, six stages
    ("bitmap", 1088, 33_333, 224),     # seventeen words: odd, five K-blocks, ring of four stages
    ("bitmap", 1536, 40_000, 300),     # six K-blocks: resident once
    ("sign", 2112, 33_333, 130),       # thirty-three words, nine K-blocks
    ("multibucket", 128, 40_001, 9),   # eight words
    ("multibucket", 832, 33_000, 260), # fifty-two words, two query tiles, ring
])
def test_fp4_filter_equals_popcount_scan(monkeypatch, kind, dim, n, nq):
    docs = ob.synth_docs(dim + n, n, dim)
    docs[5::97] = docs[4]  # exact ties across tiles
    queries, _ = ob.synth_queries(dim + n, n, nq, dim)
    ix = _index(kind, dim, docs)
    monkeypatch.setenv("OVB_FASTSCAN_FILTER", "1")
    monkeypatch.setenv("OVB_BITMAP_TC", "1")
    got = _top_m(ix, kind, queries, 200)
    monkeypatch.setenv("OVB_BITMAP_TC", "0")
    assert np.array_equal(got, _top_m(ix, kind, queries, 200))
