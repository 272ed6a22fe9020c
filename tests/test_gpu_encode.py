"""The binned rank transform of the device encoders at the edges of its forms:
row lengths around every template's limit (one warp up to 1,024, four warps
up to 4,096, sorted above), and rows that bin well, straddle bucket
boundaries with ties, crowd one bin, or are constant.  Codes are compared
byte for byte with the oracle's."""
import numpy as np
import pytest

import ordvec_b200 as ob
from ordvec_b200._lib import OrdvecError

pytestmark = pytest.mark.gpu

KINDS = ["plain", "ties", "outlier", "sparse", "constant", "denormal", "wide"]


def _docs(dim, n, seed):
    """Rows of every kind in turn, so that the rows of one CTA take different routes."""
    rng = np.random.default_rng(seed)
    d = rng.standard_normal((n, dim)).astype(np.float32)
    for i in range(n):
        kind = KINDS[i % len(KINDS)]
        if kind == "ties":
            d[i] = np.round(d[i] * 4) / 4
        elif kind == "outlier":
            d[i, i % dim] = 1e30
        elif kind == "sparse":
            d[i, rng.random(dim) < 0.7] = 0.0
            d[i, ::3] *= -0.0
        elif kind == "constant":
            d[i] = -0.0 if i % 2 else 3.5
        elif kind == "denormal":
            d[i] *= np.float32(1e-39)
        elif kind == "wide":
            d[i] = d[i] / np.abs(d[i]).max() * np.float32(3.0e38)
    return d


@pytest.mark.parametrize("dim", [2, 31, 256, 257, 384, 385, 512, 513, 768, 769, 1024, 1025, 2048, 2049, 4096, 4097])
def test_rank_rows(orc, dim):
    docs = _docs(dim, 30, dim)
    rk = ob.Rank(dim)
    rk.add(docs[:13])
    rk.add(docs[13:])
    assert np.array_equal(rk.payload().view(np.uint16), orc.rank_encode(docs, dim))


@pytest.mark.parametrize("dim", [64, 240, 256, 272, 384, 400, 512, 528, 768, 784, 1024, 1040, 2048, 4096, 4112])
def test_bucket_rows(orc, dim):
    docs = _docs(dim, 43, 7 * dim)
    for bits in (1, 2, 4):
        rq = ob.RankQuant(dim, bits)
        rq.add(docs)
        assert np.array_equal(rq.payload(), orc.rankquant_encode(docs, dim, bits)), bits
    fs = ob.RankQuantFastscan(dim)
    fs.add(docs)
    assert np.array_equal(fs.payload(), orc.fastscan_pack(docs, dim))
    if dim % 64 == 0:
        for n_top in (1, dim // 4, dim - 1):
            bm = ob.Bitmap(dim, n_top)
            bm.add(docs)
            assert np.array_equal(bm.payload().view(np.uint64), orc.bitmap_encode(docs, dim, n_top)), n_top
        for bits in (1, 4):
            mb = ob.MultiBucketBitmap(dim, bits)
            mb.add(docs)
            assert np.array_equal(mb.payload().view(np.uint64), orc.multibucket_encode(docs, dim, bits)), bits
        sb = ob.SignBitmap(dim)
        sb.add(docs)
        assert np.array_equal(sb.payload().view(np.uint64), orc.sign_encode(docs, dim))


@pytest.mark.parametrize("dim", [64, 320, 1024, 2048])
def test_bitmap_query_ties_take_the_lower_index(orc, dim):
    n_top = dim // 4
    qs = _docs(dim, 21, 3 * dim)
    docs = np.random.default_rng(dim).standard_normal((300, dim)).astype(np.float32)
    words = orc.bitmap_encode(docs, dim, n_top)
    bm = ob.Bitmap(dim, n_top)
    bm.add(docs)
    got = np.stack(bm.top_m_candidates_batched(qs, 100))
    want = np.stack([orc.bitmap_top_m(words, 300, dim, n_top, q, 100) for q in qs])
    assert np.array_equal(got, want)


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("dim", [64, 1024, 2048, 8192])
def test_device_add_refuses_non_finite_rows_and_keeps_the_index(orc, bad, dim):
    import torch

    docs = _docs(dim, 50, dim + 1)
    worse = docs.copy()
    worse[37, dim - 1] = bad
    good, spoilt = torch.from_numpy(docs).cuda(), torch.from_numpy(worse).cuda()
    torch.cuda.synchronize()
    for make, want in ((lambda: ob.RankQuant(dim, 2), lambda x: orc.rankquant_encode(x, dim, 2)),
                       (lambda: ob.SignBitmap(dim), lambda x: orc.sign_encode(x, dim).view(np.uint8).reshape(-1)),
                       (lambda: ob.RankQuantFastscan(dim), lambda x: orc.fastscan_pack(x, dim))):
        ix = make()
        with pytest.raises(OrdvecError):
            ix.add_device(spoilt.data_ptr(), 50)
        assert len(ix) == 0
        ix.add_device(good.data_ptr(), 41)
        with pytest.raises(OrdvecError):
            ix.add_device(spoilt.data_ptr(), 50)
        assert len(ix) == 41
        assert np.array_equal(ix.payload(), np.asarray(want(docs[:41])).view(np.uint8).reshape(-1))
