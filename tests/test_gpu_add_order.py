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
