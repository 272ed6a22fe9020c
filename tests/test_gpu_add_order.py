"""Adds while the default stream has work queued: what an add clears, copies and encodes
is ordered among itself, whatever that stream does and when."""
import numpy as np
import pytest

import ordvec_b200 as ob
from ordvec_b200._lib import OrdvecError

pytestmark = pytest.mark.gpu

DIM, N = 256, 1000


def _busy(torch):
    torch.cuda._sleep(200_000_000)  # about 0.1 s of the default stream


def test_fastscan_rows_survive_the_padding_clear(orc):
    torch = pytest.importorskip("torch")
    docs = np.random.default_rng(1).standard_normal((N, DIM)).astype(np.float32)
    good = torch.from_numpy(docs).cuda()
    torch.cuda.synchronize()
    fs = ob.RankQuantFastscan(DIM)
    _busy(torch)
    fs.add_device(good.data_ptr(), N)
    torch.cuda.synchronize()
    assert np.array_equal(fs.payload(), orc.fastscan_pack(docs, DIM))


def test_fastscan_rows_survive_the_clear_of_a_refused_add(orc):
    torch = pytest.importorskip("torch")
    docs = np.random.default_rng(2).standard_normal((N, DIM)).astype(np.float32)
    good = torch.from_numpy(docs).cuda()
    bad = good.clone()
    bad[N - 1, 3] = float("nan")
    torch.cuda.synchronize()
    fs = ob.RankQuantFastscan(DIM)
    _busy(torch)
    with pytest.raises(OrdvecError):
        fs.add_device(bad.data_ptr(), N)
    fs.add_device(good.data_ptr(), N - 17)  # a last block that is not full
    torch.cuda.synchronize()
    assert np.array_equal(fs.payload(), orc.fastscan_pack(docs[:N - 17], DIM))


def test_rows_survive_growth(orc):
    torch = pytest.importorskip("torch")
    docs = np.random.default_rng(3).standard_normal((N, DIM)).astype(np.float32)
    good = torch.from_numpy(docs).cuda()
    torch.cuda.synchronize()
    rq = ob.RankQuant(DIM, 4)
    at = 0
    for rows in (100, 101, 299, 500):
        _busy(torch)
        rq.add_device(good[at:].data_ptr(), rows)
        at += rows
    torch.cuda.synchronize()
    assert np.array_equal(rq.payload(), orc.rankquant_encode(docs, DIM, 4))


@pytest.mark.parametrize("make", [lambda: ob.RankQuant(DIM, 4), lambda: ob.RankQuantFastscan(DIM),
                                  lambda: ob.SignBitmap(DIM)])
def test_a_refused_add_takes_no_memory(make):
    torch = pytest.importorskip("torch")
    n = 2_000_000
    bad = torch.randn(n, DIM, device="cuda")
    bad[n // 2, 7] = float("inf")
    small = torch.randn(64, DIM, device="cuda")
    torch.cuda.synchronize()
    warm = make()  # what a first add of this thread allocates
    warm.add_device(small.data_ptr(), 64)
    ix = make()
    if not isinstance(ix, ob.RankQuantFastscan):
        ix.add_device(small.data_ptr(), 64)
    had, before = ix.payload(), torch.cuda.mem_get_info()[0]
    with pytest.raises(OrdvecError) as e:
        ix.add_device(bad.data_ptr(), n)
    assert e.value.status == 2 and "non-finite" in str(e.value)
    assert torch.cuda.mem_get_info()[0] == before
    assert np.array_equal(ix.payload(), had)


def test_non_finite_rows_are_reported_before_a_lack_of_memory():
    """Rows for which no buffer can be had (the rest of the device is held): refused as
    before for what they are, and by the allocation only when they are finite."""
    torch = pytest.importorskip("torch")
    n = 1_000_000
    rows = torch.randn(n, DIM, device="cuda")
    ix = ob.Rank(DIM)  # 512 MB of codes
    ix.add_device(rows.data_ptr(), 64)
    torch.cuda.synchronize()
    held = torch.empty(max(0, torch.cuda.mem_get_info()[0] - (256 << 20)), dtype=torch.uint8, device="cuda")
    with pytest.raises(OrdvecError) as e:
        ix.add_device(rows.data_ptr(), n)
    assert "non-finite" not in str(e.value)
    rows[5, 5] = float("nan")
    torch.cuda.synchronize()
    with pytest.raises(OrdvecError) as e:
        ix.add_device(rows.data_ptr(), n)
    assert e.value.status == 2 and "non-finite" in str(e.value)
    assert len(ix) == 64
    del held
    torch.cuda.empty_cache()
