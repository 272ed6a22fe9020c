"""Integer row scores on the CUDA cores, in front of the FP64 rescoring: the bits of the
FP64 scan and rerank, for every code width, rows of one 16-byte piece, of a partial and of
several staged chunks, one to five queries, ties across the cut, special queries, captured
streams and both sides of the rules on sizes."""
import numpy as np
import pytest

import ordvec_b200 as ob

pytestmark = pytest.mark.gpu


def _both(monkeypatch, call):
    out = []
    for form in "01":
        monkeypatch.setenv("OVB_ROW_SCORES", form)
        monkeypatch.setenv("OVB_RANK_TC", "0")
        out.append(call())
    monkeypatch.delenv("OVB_ROW_SCORES")
    monkeypatch.delenv("OVB_RANK_TC")
    out.append(call())
    for got in out[1:]:
        assert np.array_equal(got.indices, out[0].indices)
        assert np.array_equal(got.scores.view(np.uint32), out[0].scores.view(np.uint32))


@pytest.mark.parametrize("nq", [1, 2, 3, 5])
@pytest.mark.parametrize("bits,dim", [(1, 128), (1, 2176), (2, 64), (2, 1088), (4, 64), (4, 576), (4, 1024)])
def test_full_scans_agree_bit_for_bit(monkeypatch, bits, dim, nq):
    n = 4099  # a last warp of three rows
    rng = np.random.default_rng(bits * dim + nq)
    docs = rng.standard_normal((n, dim)).astype(np.float32)
    docs[2000:2300] = docs[17]  # more equal documents than the margin test lets through
    q = rng.standard_normal((nq, dim)).astype(np.float32)
    q[nq - 1] = docs[17] if nq != 2 else 0.0
    ix = ob.RankQuant(dim, bits)
    ix.add(docs)
    for k in (1, 100, 400):
        _both(monkeypatch, lambda: ix.search_asymmetric(q, k))
        _both(monkeypatch, lambda: ix.search(q, k))


@pytest.mark.parametrize("bits,dim", [(1, 1024), (2, 64), (2, 1088), (4, 1024)])
def test_two_stage_agrees_bit_for_bit(monkeypatch, bits, dim):
    n, nq = 5003, 9
    rng = np.random.default_rng(dim + bits)
    docs = rng.standard_normal((n, dim)).astype(np.float32)
    docs[100:400] = docs[50]
    q = (docs[rng.integers(0, n, nq)] + 0.3 * rng.standard_normal((nq, dim))).astype(np.float32)
    q[4] = docs[50]
    rq, sb = ob.RankQuant(dim, bits), ob.SignBitmap(dim)
    rq.add(docs)
    sb.add(docs)
    for m, k in ((1000, 10), (2500, 200), (333, 1)):
        _both(monkeypatch, lambda: ob.two_stage_search(rq, sb, q, m, k))


def test_both_sides_of_the_size_rules(monkeypatch):
    """8e8 = 1 x n x 1,024 x 2 at n = 390,625; candidates: 5e8 = nq x 1,000 x 1,024 x 2."""
    dim, n = 1024, 390_700
    docs = ob.synth_docs(3, n, dim)
    rq, sb = ob.RankQuant(dim, 2), ob.SignBitmap(dim)
    q, _ = ob.synth_queries(3, n, 245, dim)
    rq.add(docs[:390_600])
    _both(monkeypatch, lambda: rq.search_asymmetric(q[:1], 10))
    rq.add(docs[390_600:])
    _both(monkeypatch, lambda: rq.search_asymmetric(q[:1], 10))
    sb.add(docs)
    for nq in (244, 245):
        _both(monkeypatch, lambda: ob.two_stage_search(rq, sb, q[:nq], 1000, 10))


@pytest.mark.parametrize("nq", [2, 8])
@pytest.mark.parametrize("kind", ["rankquant", "rank"])
def test_capture_after_an_eager_call(kind, nq):
    """A captured search needs no buffer that the eager search before it did not size."""
    torch = pytest.importorskip("torch")
    dim, n, k = 512, 400_000, 10
    docs = ob.synth_docs(9, n, dim)
    q = torch.from_numpy(ob.synth_queries(9, n, nq, dim)[0]).cuda()
    ix = ob.RankQuant(dim, 4) if kind == "rankquant" else ob.Rank(dim)
    ix.add(docs)
    s = torch.empty(nq * k, device="cuda")
    i = torch.empty(nq * k, dtype=torch.int64, device="cuda")
    side = torch.cuda.Stream()
    for asym in (True, False):
        call = lambda: ob.search_device(ix, q.data_ptr(), nq, k, s.data_ptr(), i.data_ptr(), side.cuda_stream,  # noqa: E731
                                        asymmetric=asym)
        call()
        side.synchronize()
        want = s.clone(), i.clone()
        s.zero_(), i.zero_()
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=side):
            call()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(i, want[1]) and torch.equal(s, want[0])


def test_an_equal_run_across_the_cut(monkeypatch):
    """Symmetric scores tie by the thousand: the order is (score, id) and no fallback is
    needed; asymmetric equal documents take it."""
    dim, n = 128, 300_000
    docs = np.random.default_rng(2).standard_normal((n, dim)).astype(np.float32)
    docs[1000:5000] = docs[3]
    q = np.concatenate([docs[3:4], docs[70:71]])
    for bits in (1, 4):
        ix = ob.RankQuant(dim, bits)
        ix.add(docs)
        _both(monkeypatch, lambda: ix.search(q, 64))
        _both(monkeypatch, lambda: ix.search_asymmetric(q, 64))
        batch = np.concatenate([q] * 40)  # the tensor-core forms
        many = ix.search(batch, 64)
        one = ix.search(q, 64)
        assert np.array_equal(many.indices.reshape(80, -1)[:2], one.indices.reshape(2, -1))
