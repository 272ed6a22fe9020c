"""Query tiles of the integer MMAs across CTA pairs, whose N is a multiple of 32: batch
sizes at and around the edges of a tile for Rank byte planes (three columns a query),
int8 bitmaps and FastScan.  Ids, ties included, and score bits equal the CUDA cores'."""
import numpy as np
import pytest

import ordvec_b200 as ob

pytestmark = pytest.mark.gpu

N, DIM = 33_100, 192


@pytest.fixture(scope="module")
def data():
    docs = ob.synth_docs(11, N, DIM)
    docs[7::301] = docs[6]
    return docs, ob.synth_queries(11, N, 260, DIM)[0]


@pytest.mark.parametrize("nq", [1, 2, 16, 17, 32, 33, 48, 49, 64, 65, 96, 97])
def test_rank(monkeypatch, data, nq):
    docs, q = data
    rk = ob.Rank(DIM)
    rk.add(docs)
    for search in (rk.search, rk.search_asymmetric):
        out = []
        for tc in "01":
            monkeypatch.setenv("OVB_RANK_TC", tc)
            out.append(search(q[:nq], 20))
        assert np.array_equal(out[0].indices, out[1].indices)
        assert np.array_equal(out[0].scores.view(np.uint32), out[1].scores.view(np.uint32))


@pytest.mark.parametrize("nq", [1, 15, 17, 32, 33, 48, 49, 223, 225, 255, 256, 257])
def test_int8_bitmaps_and_fastscan(monkeypatch, data, nq):
    docs, q = data
    sb, bm, fs = ob.SignBitmap(DIM), ob.Bitmap(DIM, 48), ob.RankQuantFastscan(DIM)
    for ix in (sb, bm, fs):
        ix.add(docs)
    monkeypatch.setenv("OVB_TC_FORM", "pair")
    monkeypatch.setenv("OVB_BITMAP_FP4", "0")
    out = []
    for tc in "01":
        monkeypatch.setenv("OVB_BITMAP_TC", tc)
        monkeypatch.setenv("OVB_FASTSCAN_TC", tc)
        out.append([np.stack(ix.top_m_candidates_batched(q[:nq], 300)) for ix in (sb, bm)] +
                   [fs.search(q[:nq], 50).indices])
    for want, got in zip(*out):
        assert np.array_equal(got, want)
