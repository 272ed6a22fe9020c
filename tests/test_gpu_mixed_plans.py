"""A mixed plan whose replayed graph is followed by the exact pipeline in the same
workspace: a batch that keeps too few documents at its sampled thresholds, but passes
the margin test with the plan's own candidate count, moves the buffer of the candidate
rows that the graph writes its thresholds to.  The next replays answer as before and
leave memory that was allocated in between alone."""
import numpy as np
import pytest

import ordvec_b200 as ob

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bits", [1, 4])
def test_replays_after_a_batch_below_its_thresholds(monkeypatch, bits):
    torch = pytest.importorskip("torch")
    n, dim, nq, k = 150_000, 256, 400, 100
    rng = np.random.default_rng(bits)
    docs = rng.standard_normal((n, dim)).astype(np.float32)
    near = rng.standard_normal(dim).astype(np.float32)
    # every 32nd block of 32 documents is in the sample: two of them hold all that is near
    # this query, more than the rank of the threshold (35) and fewer than the candidates (200)
    for first in (0, 1024):
        docs[first:first + 32] = near + 0.3 * rng.standard_normal((32, dim)).astype(np.float32)
    rq = ob.RankQuant(dim, bits)
    rq.add(docs)
    good = (docs[rng.integers(2048, n, nq)] + 0.5 * rng.standard_normal((nq, dim))).astype(np.float32)
    low = good.copy()
    low[7] = near
    which, ks = np.zeros(nq, np.uint32), np.full(nq, k, np.uint32)
    call = lambda q: ob.search_mixed([rq], which, ks, q)  # noqa: E731
    monkeypatch.setenv("OVB_MIXED_GRAPH", "0")
    want = {id(q): call(q) for q in (good, low)}
    monkeypatch.delenv("OVB_MIXED_GRAPH")
    for step, q in enumerate((good, good, low, good, low, good)):  # tune and capture, replay, fail, ...
        got = call(q)
        if step == 2:  # what the freed buffer's memory may become
            held = [torch.full((1 << 19,), 7, dtype=torch.int32, device="cuda") for _ in range(8)]
        assert np.array_equal(got.indices, want[id(q)].indices), step
        assert np.array_equal(got.scores.view(np.uint32), want[id(q)].scores.view(np.uint32)), step
    info = ob.mixed_plan_info(rq, nq, k)
    assert info["candidates"] == 200  # the margin test passed with the plan's own count
    assert info["replays"] == 5
    torch.cuda.synchronize()
    assert all(bool((h == 7).all()) for h in held)
