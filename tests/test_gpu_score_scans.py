"""The integer candidate scans (RankQuant codes in 16-bit fixed point, Rank rows as
byte planes) at the edges of their tiles: partial query tiles and several of them,
rows that end inside a K-block, rows of whole 16-byte pieces and of 8-byte ones,
partial last document tiles, and queries the bound cannot serve (constant, zero,
one large coordinate).  The searches are exact: ids, ties included, and score bits
equal the forms that score every document on the CUDA cores."""
import numpy as np
import pytest

import ordvec_b200 as ob

pytestmark = pytest.mark.gpu


def _data(dim, n, nq, seed):
    docs = ob.synth_docs(seed, n, dim)
    docs[3::501] = docs[2]  # exact ties
    queries, _ = ob.synth_queries(seed, n, nq, dim)
    return docs, queries


def _both(monkeypatch, run):
    out = []
    for tc in ("1", "0"):
        monkeypatch.setenv("OVB_RANK_TC", tc)
        out.append(run())
    a, b = out
    assert np.array_equal(a.indices, b.indices)
    assert np.array_equal(a.scores.view(np.uint32), b.scores.view(np.uint32))


@pytest.mark.parametrize("bits,dim,n,nq", [
    (1, 64, 40_001, 5),        # half a K-block, rows of 8 bytes
    (1, 320, 33_001, 130),     # rows of 40 bytes, two query tiles
    (1, 1024, 33_333, 17),
    (2, 192, 40_001, 33),      # rows of 48 bytes, one and a half K-blocks
    (2, 768, 50_000, 129),
    (4, 64, 33_000, 16),
    (4, 832, 33_333, 300),     # six and a half K-blocks, three query tiles
    (4, 1024, 70_001, 1),
])
def test_rankquant_fixed_point_scan(monkeypatch, bits, dim, n, nq):
    docs, queries = _data(dim, n, nq, dim + bits)
    if nq > 4:
        queries[1] = 0.0
        queries[2] = 1.0
        queries[3, 7] = 1e6
    rq = ob.RankQuant(dim, bits)
    rq.add(docs)
    _both(monkeypatch, lambda: rq.search_asymmetric(queries, 20))
    _both(monkeypatch, lambda: rq.search(queries, 20))


@pytest.mark.parametrize("dim,n,nq", [
    (64, 40_001, 3),           # one K-block
    (72, 33_001, 65),          # rows of 144 bytes: a K-block and 16 bytes; two query tiles
    (200, 33_333, 16),
    (768, 45_000, 64),
    (1024, 33_333, 19),
    (1000, 33_333, 130),       # three query tiles, a partial last K-block
    (2048, 33_000, 7),         # the longest rows of the form
])
def test_rank_byte_planes(monkeypatch, dim, n, nq):
    docs, queries = _data(dim, n, nq, dim)
    if nq > 6:
        queries[1] = 0.0
        queries[2] = -2.5
        queries[3, 5] = 1e6
    rk = ob.Rank(dim)
    rk.add(docs)
    _both(monkeypatch, lambda: rk.search(queries, 30))
    _both(monkeypatch, lambda: rk.search_asymmetric(queries, 30))


def test_rank_search_under_capture_has_no_host_read():
    """A capturing stream keeps the forms without a host-side flag."""
    import torch

    dim, n, nq, k = 256, 200_000, 32, 10
    docs, queries = _data(dim, n, nq, 5)
    rk, rq = ob.Rank(dim), ob.RankQuant(dim, 4)
    rk.add(docs)
    rq.add(docs)
    q = torch.from_numpy(queries).cuda()
    stream = torch.cuda.Stream()
    for ix in (rk, rq):
        s, i = torch.empty(nq * k, device="cuda"), torch.empty(nq * k, dtype=torch.int64, device="cuda")
        call = lambda: ob.search_device(ix, q.data_ptr(), nq, k, s.data_ptr(), i.data_ptr(), stream.cuda_stream,
                                        asymmetric=True)
        with pytest.MonkeyPatch.context() as m:  # size the buffers of the captured form
            m.setenv("OVB_RANK_TC", "0")
            call()
        torch.cuda.synchronize()
        want = i.clone()
        i.zero_()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=stream):
            call()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(i, want)
        call()
        torch.cuda.synchronize()
        assert torch.equal(i, want)
