"""Queries whose integer candidates are not known to hold their top k are scored again
exactly, and only they: batches in which none, a few and all of the queries meet more
equal documents across the cut than the candidates hold, for every form that has the
exact pass behind it, on both sides of the limit for results in pinned memory, through
device pointers, and with the key matrix in chunks.  Ids and score bits equal the forms
that score every document exactly."""
import os
import subprocess
import sys

import numpy as np
import pytest

import ordvec_b200 as ob

pytestmark = pytest.mark.gpu

DIM = 256


def _docs(n, equal, seed=5):
    docs = np.random.default_rng(seed).standard_normal((n, DIM)).astype(np.float32)
    docs[n // 3:n // 3 + equal // 2] = docs[9]
    docs[-(equal - equal // 2):] = docs[9]
    return docs


def _queries(docs, nq, which):
    """Noisy documents; those listed in `which` are the equal one, the last of them zero."""
    rng = np.random.default_rng(nq)
    q = (docs[100 + rng.integers(0, 1000, nq)] + 0.3 * rng.standard_normal((nq, DIM))).astype(np.float32)
    for i in which:
        q[i] = docs[9] + 1e-4 * rng.standard_normal(DIM)
    if len(which) > 1:
        q[which[-1]] = 0.0
    return q


def _which(nq, some):
    return {"none": [], "some": sorted({0, nq // 2, nq - 1}), "all": list(range(nq))}[some]


def _exact(monkeypatch, call):
    with monkeypatch.context() as m:
        m.setenv("OVB_RANK_TC", "0")
        m.setenv("OVB_ROW_SCORES", "0")
        return call()


def _same(got, want):
    assert np.array_equal(got.indices, want.indices)
    assert np.array_equal(got.scores.view(np.uint32), want.scores.view(np.uint32))


@pytest.mark.parametrize("some", ["none", "some", "all"])
@pytest.mark.parametrize("bits,nq", [(4, 1), (4, 4), (2, 17), (2, 63)])  # row scores; the filter
def test_rankquant(monkeypatch, bits, nq, some):
    docs = _docs(1_000_000 if nq == 1 else 300_000, 1000)
    rq = ob.RankQuant(DIM, bits)
    rq.add(docs)
    q = _queries(docs, nq, _which(nq, some))
    for k in (10, 300):  # 63 x 300 results are beyond pinned memory
        call = lambda: rq.search_asymmetric(q, k)  # noqa: E731
        _same(call(), _exact(monkeypatch, call))
    call = lambda: rq.search(q, 10)  # noqa: E731
    _same(call(), _exact(monkeypatch, call))


@pytest.mark.parametrize("some", ["none", "some", "all"])
@pytest.mark.parametrize("nq", [13, 64])
def test_rank(monkeypatch, nq, some):
    docs = _docs(300_000, 1000)
    rk = ob.Rank(DIM)
    rk.add(docs)
    q = _queries(docs, nq, _which(nq, some))
    for k in (10, 300):
        for search in (rk.search, rk.search_asymmetric):
            call = lambda: search(q, k)  # noqa: E731
            _same(call(), _exact(monkeypatch, call))


@pytest.mark.parametrize("some", ["none", "some", "all"])
@pytest.mark.parametrize("bits,nq", [(4, 520), (4, 1000)])  # 1,024 bits a row
def test_two_stage_rerank(monkeypatch, bits, nq, some):
    docs = _docs(20_000, 1000)
    rq, sb = ob.RankQuant(DIM, bits), ob.SignBitmap(DIM)
    rq.add(docs)
    sb.add(docs)
    q = _queries(docs, nq, _which(nq, some))
    call = lambda: ob.two_stage_search(rq, sb, q, 1000, 20)  # noqa: E731
    _same(call(), _exact(monkeypatch, call))


@pytest.mark.parametrize("kind", ["rankquant", "rank"])
def test_device_results(monkeypatch, kind):
    torch = pytest.importorskip("torch")
    docs, nq, k = _docs(300_000, 1000), 24, 50
    ix = ob.RankQuant(DIM, 2) if kind == "rankquant" else ob.Rank(DIM)
    ix.add(docs)
    q = _queries(docs, nq, _which(nq, "some"))
    d = torch.from_numpy(q).cuda()
    s, i = torch.empty(nq * k, device="cuda"), torch.empty(nq * k, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    ob.search_device(ix, d.data_ptr(), nq, k, s.data_ptr(), i.data_ptr(), torch.cuda.current_stream().cuda_stream,
                     asymmetric=True)
    torch.cuda.synchronize()
    want = _exact(monkeypatch, lambda: ix.search_asymmetric(q, k))
    assert np.array_equal(i.cpu().numpy(), want.indices)
    assert np.array_equal(s.cpu().numpy().view(np.uint32), want.scores.view(np.uint32))


def test_key_matrix_in_chunks():
    """Two queries of keys a chunk (the budget is read once a process)."""
    if "OVB_KEYS_BUDGET_MB" in os.environ:
        pytest.skip("runs the other tests under a small budget itself")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    r = subprocess.run([sys.executable, "-m", "pytest", os.path.abspath(__file__), "-x", "-q", "-m", "gpu", "-k",
                        "test_rank or test_device"], cwd=root, env=dict(os.environ, OVB_KEYS_BUDGET_MB="3"),
                       capture_output=True, text=True, timeout=600)
    assert r.returncode == 0, r.stdout[-3000:] + r.stderr[-2000:]
