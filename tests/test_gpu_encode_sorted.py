"""The sorted form of the device encoders, which takes the rows that bin badly (half of the
values equal, all values of two kinds, tails that crowd the rest into a few bins) and all rows
beyond 4,096: a warp's sort, a CTA's with 1 to 32 keys a thread, and every emission, byte for
byte against the oracle."""
import numpy as np
import pytest

import ordvec_b200 as ob

pytestmark = pytest.mark.gpu


def _docs(dim, n):
    rng = np.random.default_rng(dim)
    d = rng.standard_normal((n, dim)).astype(np.float32)
    d[0::4] = np.maximum(d[0::4], 0)
    d[1::4] = d[1::4] > 0
    d[2::4] = d[2::4] ** 9
    return d  # every fourth row bins well


@pytest.mark.parametrize("dim", [2, 33, 200, 256, 257, 512, 768, 1000, 1024, 2048, 4096, 4098, 8192, 8194, 16384])
def test_rank_rows(orc, dim):
    docs = _docs(dim, 21)
    rk = ob.Rank(dim)
    rk.add(docs)
    assert np.array_equal(rk.payload().view(np.uint16), orc.rank_encode(docs, dim))


@pytest.mark.parametrize("dim", [64, 128, 256, 320, 512, 576, 768, 1024, 1088, 2048, 4096, 8192, 16384])
def test_bucket_rows(orc, dim):
    docs = _docs(dim, 21)
    for bits in (1, 2, 4):
        rq = ob.RankQuant(dim, bits)
        rq.add(docs)
        assert np.array_equal(rq.payload(), orc.rankquant_encode(docs, dim, bits)), bits
        mb = ob.MultiBucketBitmap(dim, bits)
        mb.add(docs)
        assert np.array_equal(mb.payload().view(np.uint64), orc.multibucket_encode(docs, dim, bits)), bits
    fs, bm = ob.RankQuantFastscan(dim), ob.Bitmap(dim, dim // 4)
    fs.add(docs)
    bm.add(docs)
    assert np.array_equal(fs.payload(), orc.fastscan_pack(docs, dim))
    words = orc.bitmap_encode(docs, dim, dim // 4)
    assert np.array_equal(bm.payload().view(np.uint64), words)
    got = np.stack(bm.top_m_candidates_batched(docs, 7))  # the queries' bits: descending, ties to the lower index
    want = np.stack([orc.bitmap_top_m(words, len(docs), dim, dim // 4, q, 7) for q in docs])
    assert np.array_equal(got, want)


@pytest.mark.parametrize("n", [1, 591, 592, 593])
@pytest.mark.parametrize("dim", [128, 129, 256, 257, 512, 520, 1024])
def test_ranks_of_a_batch(orc, dim, n):
    """Both sides of the number of rows from which full ranks are binned."""
    docs = _docs(dim, n)
    rk = ob.Rank(dim)
    rk.add(docs)
    assert np.array_equal(rk.payload().view(np.uint16), orc.rank_encode(docs, dim))
