"""Workloads of the compressed-scan path, through the package's public calls.

Five kinds of pass, each as a user's program makes it:

* ``two_stage``  candidate generation (SignBitmap, Bitmap, FastScan or MultiBucketBitmap) and
                 RankQuant rerank over indices that stay on the device; queries either in host
                 memory (``two_stage_search``) or on the device (``two_stage_search_device``)
* ``full``       exhaustive RankQuant search, asymmetric or symmetric
* ``rank``       exhaustive search of the full-precision Rank index, symmetric or asymmetric
* ``mixed``      one call for queries with their own index (bits 1, 2, 4) and k
* ``ingest``     documents that are on the device (an embedding model's output) become indices,
                 which answer a first batch of queries: an index that lives for one session, or a
                 shard that is rebuilt

Documents are a mixture of 256 Gaussian clusters (unit-norm centres, sigma 0.3 per coordinate,
normalised), queries perturbed documents (sigma 0.1, normalised): the corpus of the repository's own
benchmark.
"""
import math

import numpy as np
import torch

import ordvec_b200 as ob

CHUNK_BYTES = 1 << 29  # documents are made and encoded this many bytes at a time


def listed():
    return [
        # one query per call on a small sign-bitmap corpus: the smallest call, an interactive lookup
        dict(name="sign_b1_one", op="two_stage", stage1="sign", host=True, n=100_000, dim=1024, bits=1, nq=1, m=320, k=10),
        # one query per call, FastScan candidates: the plain two-stage configuration
        dict(name="fastscan_one", op="two_stage", stage1="fastscan", host=True, n=171_332, dim=1024, bits=2, nq=1, m=1000, k=10),
        # one query per call over millions of documents (ragged count): an interactive search of a large corpus
        dict(name="bitmap_one_5m", op="two_stage", stage1="bitmap", host=True, n=5_000_003, dim=768, bits=2, nq=1, m=2000, k=100),
        # a batch over the plain two-stage configuration: offline evaluation of a query set
        dict(name="fastscan_batch", op="two_stage", stage1="fastscan", host=False, n=171_332, dim=1024, bits=2, nq=1000, m=1000, k=10),
        # the large-corpus configuration: batches of 1,024 queries over 10M documents
        dict(name="bitmap_batch_10m", op="two_stage", stage1="bitmap", host=False, n=10_000_000, dim=768, bits=2, nq=1024, m=2000, k=100),
        # multi-bucket candidates, an ordinary batch over a mid-size corpus
        dict(name="multibucket_batch", op="two_stage", stage1="multibucket", host=False, n=1_000_000, dim=768, bits=2, nq=256, m=2000, k=100),
        # one request of the serving loop: a ragged handful of queries, 4-bit codes, default policy (m = 0)
        dict(name="sign_serving", op="two_stage", stage1="sign", host=True, n=1_000_000, dim=1024, bits=4, nq=61, m=0, k=50),
        # an exhaustive 2-bit search of one query: recall checks, small corpora without candidates
        dict(name="rankquant_one", op="full", symmetric=False, host=True, n=1_000_000, dim=768, bits=2, nq=1, k=10),
        # queries of mixed bits and k against three indices in one call
        dict(name="mixed_batch", op="mixed", n=1_000_000, dim=1024, nq=4096, k=100),
        # full-precision rank search, a batch on the device
        dict(name="rank_sym_batch", op="rank", asymmetric=False, host=False, n=1_000_000, dim=768, nq=64, k=100),
        # full-precision rank search against float queries, a small ragged host batch
        dict(name="rank_asym_small", op="rank", asymmetric=True, host=True, n=250_007, dim=1024, nq=19, k=50),
        # documents on the device become a Bitmap and a RankQuant index that answer a first batch
        dict(name="ingest", op="ingest", n=120_000, dim=768, bits=2, nq=64, m=1000, k=100),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """Another case of the same kinds; sizes log-uniform over the range the listed ones span."""
    op = rng.choice(["two_stage", "two_stage", "two_stage", "full", "rank", "mixed", "ingest"])
    n = _log(rng, 30_000, 4_000_000)
    nq = 1 if rng.random() < 0.3 else _log(rng, 2, 1024)
    host = rng.random() < 0.5
    k = _log(rng, 5, 100)
    if op == "two_stage":
        stage1 = rng.choice(["sign", "bitmap", "fastscan", "multibucket"])
        dim = rng.choice([300, 384, 768, 1000, 1024]) if stage1 == "fastscan" else rng.choice([256, 384, 512, 768, 1024])
        bits = 2 if stage1 in ("fastscan", "multibucket") else rng.choice([1, 2, 4])
        if stage1 == "multibucket":
            n = min(n, 1_000_000)
        m = 0 if rng.random() < 0.25 else _log(rng, 200, 2000)
        return dict(op=op, stage1=stage1, host=host, n=n, dim=dim, bits=bits, nq=nq, m=m, k=k)
    if op == "full":
        dim = rng.choice([256, 384, 768, 1024])
        return dict(op=op, symmetric=rng.random() < 0.3, host=host, n=min(n, 1_000_000), dim=dim,
                    bits=rng.choice([1, 2, 4]), nq=min(nq, 512), k=k)
    if op == "rank":
        dim = rng.choice([200, 256, 384, 768, 1024])
        return dict(op=op, asymmetric=rng.random() < 0.5, host=host, n=min(n, 1_000_000), dim=dim,
                    nq=min(nq, 64), k=k)
    if op == "mixed":
        return dict(op=op, n=min(n, 1_000_000), dim=rng.choice([256, 512, 768, 1024]), nq=_log(rng, 64, 4096), k=100)
    return dict(op=op, n=_log(rng, 10_000, 400_000), dim=rng.choice([384, 768, 1024]), bits=rng.choice([1, 2, 4]),
                nq=_log(rng, 1, 256), m=_log(rng, 200, 1000), k=k)


def _generator(seed, stream):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 1_000_003 + stream)


def _corpus(case, seed, queries):
    """Yields (first row, documents) chunk by chunk and fills `queries` with rows that it passes."""
    n, dim, nq = case["n"], case["dim"], case["nq"]
    g = _generator(seed, 1)
    centres = torch.randn(256, dim, generator=g, device="cuda")
    centres /= centres.norm(dim=1, keepdim=True)
    pick = torch.randint(n, (nq,), generator=g, device="cuda")
    step = max(32, CHUNK_BYTES // (4 * dim) // 32 * 32)
    for first in range(0, n, step):
        rows = min(step, n - first)
        docs = torch.randn(rows, dim, generator=g, device="cuda").mul_(0.3)
        docs += centres[torch.randint(256, (rows,), generator=g, device="cuda")]
        docs /= docs.norm(dim=1, keepdim=True)
        here = (pick >= first) & (pick < first + rows)
        queries[here] = docs[pick[here] - first]
        yield first, docs
    queries += 0.1 * torch.randn(nq, dim, generator=_generator(seed, 2), device="cuda")
    queries /= queries.norm(dim=1, keepdim=True)


def _n_top(case):
    return case["dim"] // 4


def _stage1(case):
    dim = case["dim"]
    return {"sign": lambda: ob.SignBitmap(dim), "bitmap": lambda: ob.Bitmap(dim, _n_top(case)),
            "fastscan": lambda: ob.RankQuantFastscan(dim), "multibucket": lambda: ob.MultiBucketBitmap(dim, 2)}[case["stage1"]]()


def prepare(case, seed):
    """The indices on the device and the queries where the call wants them."""
    op, dim, nq = case["op"], case["dim"], case["nq"]
    q = torch.empty(nq, dim, device="cuda")
    state = {"case": case}
    indices, whole = [], []
    if op == "two_stage":
        state["rq"], state["s1"] = ob.RankQuant(dim, case["bits"]), _stage1(case)
        indices = [state["rq"], state["s1"]]
        if case["stage1"] == "fastscan":  # FastScan takes its documents in one add
            indices, whole = [state["rq"]], [state["s1"]]
    elif op == "full":
        state["index"] = ob.RankQuant(dim, case["bits"])
        indices = [state["index"]]
    elif op == "rank":
        state["index"] = ob.Rank(dim)
        indices = [state["index"]]
    elif op == "mixed":
        state["indices"] = [ob.RankQuant(dim, b) for b in (1, 2, 4)]
        indices = state["indices"]
    all_docs = torch.empty(case["n"], dim, device="cuda") if whole or op == "ingest" else None
    for first, docs in _corpus(case, seed, q):
        if all_docs is not None:
            all_docs[first:first + docs.shape[0]] = docs
        torch.cuda.synchronize()
        for ix in indices:
            ix.add_device(docs.data_ptr(), docs.shape[0])
    torch.cuda.synchronize()
    for ix in whole:
        ix.add_device(all_docs.data_ptr(), case["n"])
    if op == "ingest":
        state["docs"] = all_docs
    if op == "mixed":
        r = np.random.RandomState(seed & 0x7FFFFFFF)
        state["which"] = r.randint(0, 3, nq).astype(np.uint32)
        state["k_of"] = np.array([10, 50, 100], np.uint32)[r.randint(0, 3, nq)]
        state["k_of"][0] = case["k"]
    if case.get("host", True):
        pinned = torch.empty(nq, dim, pin_memory=True)
        pinned.copy_(q)
        state["pinned"], state["q"] = pinned, pinned.numpy()
    else:
        state["q"] = q
        count = nq * min(case["k"], case["n"])
        state["scores"] = torch.empty(count, device="cuda")
        state["ids"] = torch.empty(count, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    return state


def run(state):
    """One call (for ingest: the adds and one call)."""
    c = state["case"]
    op, k = c["op"], c["k"]
    if op == "mixed":
        r = ob.search_mixed(state["indices"], state["which"], state["k_of"], state["q"])
        return [r.scores, r.indices]
    if op == "ingest":
        docs = state["docs"]
        bm, rq = ob.Bitmap(c["dim"], _n_top(c)), ob.RankQuant(c["dim"], c["bits"])
        bm.add_device(docs.data_ptr(), c["n"])
        rq.add_device(docs.data_ptr(), c["n"])
        r = ob.two_stage_search(rq, bm, state["q"], c["m"], k)
        return [r.scores, r.indices]
    if c["host"]:
        if op == "two_stage":
            r = ob.two_stage_search(state["rq"], state["s1"], state["q"], c["m"], k)
        elif op == "full":
            r = (state["index"].search if c["symmetric"] else state["index"].search_asymmetric)(state["q"], k)
        else:
            r = (state["index"].search_asymmetric if c["asymmetric"] else state["index"].search)(state["q"], k)
        return [r.scores, r.indices]
    q, s, i = state["q"].data_ptr(), state["scores"], state["ids"]
    stream = torch.cuda.current_stream().cuda_stream
    if op == "two_stage":
        ob.two_stage_search_device(state["rq"], state["s1"], q, c["nq"], c["m"], k, s.data_ptr(), i.data_ptr(), stream)
    else:
        asym = c["asymmetric"] if op == "rank" else not c["symmetric"]
        ob.search_device(state["index"], q, c["nq"], k, s.data_ptr(), i.data_ptr(), stream, asymmetric=asym)
    return [s, i]


def work(case):
    """Codes read once, queries in, results out; one multiply-add per code and query of a scan."""
    op, n, dim, nq, k = case["op"], case["n"], case["dim"], case["nq"], case["k"]
    io = nq * dim * 4 + nq * k * 12
    if op == "mixed":
        return {"bytes": n * dim * 7 // 8 + io, "flops": 2 * n * dim * nq}
    if op == "full":
        return {"bytes": n * dim * case["bits"] // 8 + io, "flops": 2 * n * dim * nq}
    if op == "rank":
        return {"bytes": n * dim * 2 + io, "flops": 2 * n * dim * nq}
    m = min(case["m"] or max(256, 32 * k), n)
    row = dim * case["bits"] // 8
    rerank = min(n, nq * m) * row
    if op == "ingest":
        return {"bytes": n * (dim * 4 + dim // 8 + row) + n * dim // 8 + rerank + io, "flops": 2 * n * dim * nq + 2 * nq * m * dim}
    code = {"sign": dim // 8, "bitmap": dim // 8, "fastscan": dim // 4, "multibucket": dim // 2}[case["stage1"]]
    return {"bytes": n * code + rerank + io, "flops": 2 * n * dim * nq + 2 * nq * m * dim}


# ---- the same results in 64 bits, without the package -----------------------------------------


def _ranks(x):
    """Ascending rank of each coordinate, equal values by index."""
    order = x.sort(dim=1, stable=True).indices
    return torch.empty_like(order).scatter_(1, order, torch.arange(x.shape[1], device=x.device).expand_as(order))


def _buckets(x, bits):
    return _ranks(x) * (1 << bits) // x.shape[1]


def _centred(x, bits):
    return _buckets(x, bits).double() - ((1 << bits) - 1) / 2


def _unit(q):
    q = q.double()
    return q / q.norm(dim=1, keepdim=True)


def _top(best, scores, k):
    """The k largest of what is held and the new columns."""
    scores = scores.topk(min(k, scores.shape[1]), dim=1).values
    best = scores if best is None else torch.cat([best, scores], 1)
    return best.topk(min(k, best.shape[1]), dim=1).values


def _one_hot(b, levels):
    return (b.unsqueeze(2) == torch.arange(levels, device=b.device)).flatten(1).float()


def _fastscan(case, q, codes):
    """Integer LUT sums and their f32 scores; the tables are quantised in f32 by definition."""
    dim = case["dim"]
    x = q.cpu().numpy()
    ss = np.stack([np.cumsum(r * r, dtype=np.float32)[-1] for r in x]).astype(np.float32)
    unit = torch.from_numpy((x * (np.float32(1) / np.sqrt(ss))[:, None]).astype(np.float32)).cuda()
    a, b = unit[:, 0::2], unit[:, 1::2]
    level = torch.tensor([-1.5, -0.5, 0.5, 1.5], device="cuda")
    v = (a[:, :, None, None] * level[:, None]) + (b[:, :, None, None] * level)
    v = v.flatten(1)
    low = v.min(1).values
    scale = 255.0 / (v.max(1).values - low).clamp_min(1e-12)
    t = (v - low[:, None]) * scale[:, None]
    lut = (t.floor() + ((t - t.floor()) >= 0.5).float()).clamp(0, 255)
    bias, inv_q = (dim // 2) * low, 1.0 / scale
    inv_norm = np.float32(1) / np.float32(math.sqrt(dim * 1.25))
    found = []
    for at in range(0, codes.shape[0], 16384):
        c = codes[at:at + 16384].long()
        acc = _one_hot(c[:, 0::2] * 4 + c[:, 1::2], 16) @ lut.T
        found.append((bias[:, None] + acc.T * inv_q[:, None]) * float(inv_norm))
    return torch.cat(found, 1)


def _two_stage(case, seed):
    n, dim, nq, bits, k = case["n"], case["dim"], case["nq"], case["bits"], case["k"]
    kind = "bitmap" if case["op"] == "ingest" else case["stage1"]
    m = min(case["m"] or max(256, 32 * k), n)
    q = torch.empty(nq, dim, device="cuda")
    codes, words = [], []
    for _, docs in _corpus(case, seed, q):
        for x in docs.split(65536):
            if kind == "sign":
                codes.append(_buckets(x, bits).to(torch.uint8))
                words.append(x > 0)
                continue
            r = _ranks(x)
            codes.append((r * (1 << bits) // dim).to(torch.uint8))
            words.append(r >= dim - _n_top(case) if kind == "bitmap" else (r * 4 // dim).to(torch.uint8))
    codes = torch.cat(codes)
    unit = _unit(q)
    norm = math.sqrt(dim * ((1 << bits) ** 2 - 1) / 12)
    qr = _ranks(q)
    if kind == "sign":
        qs = (q > 0).half() * 2 - 1
    elif kind == "bitmap":
        qs = (qr >= dim - _n_top(case)).half()
    elif kind == "multibucket":
        qs = _one_hot(qr * 4 // dim, 4).half()
    if kind == "fastscan":
        s = _fastscan(case, q, torch.cat(words))
        ids = s.sort(dim=1, descending=True, stable=True).indices[:, :m]
    else:
        # score and row in one integer, larger is better; integers of the products are exact in f32
        keys, first = None, 0
        step = max(1, (1 << 27) // nq)
        for block in words:
            for w in block.split(step):
                w = w.half() * 2 - 1 if kind == "sign" else w.half() if kind == "bitmap" else _one_hot(w, 4).half()
                s = torch.cat([a.float() @ w.float().T for a in qs.split(1024)])
                row = torch.arange(first, first + w.shape[0], device="cuda")
                first += w.shape[0]
                new = (s.long() + 2 * dim) * (1 << 32) + ((1 << 32) - 1 - row)
                keys = _top(keys, new, m)
        ids = (1 << 32) - 1 - (keys & ((1 << 32) - 1))
    out = []
    for i in range(nq):
        rows = codes[ids[i]].double() - ((1 << bits) - 1) / 2
        out.append((rows @ unit[i] / norm).sort(descending=True).values[:k])
    return [torch.cat(out), None]


def exact(case, seed):
    """Scores in 64 bits; the row ids beside them are whole numbers and have no other form."""
    op, n, dim, k = case["op"], case["n"], case["dim"], case["k"]
    if op in ("two_stage", "ingest"):
        if n * case["nq"] > 2e10:
            return None
        return _two_stage(case, seed)
    q = torch.empty(case["nq"], dim, device="cuda")
    for _ in _corpus(case, seed, q):
        pass
    widths = {"mixed": (1, 2, 4), "full": (case.get("bits"),), "rank": (0,)}[op]
    sides, best = [], []
    for bits in widths:
        if op == "rank":
            norm = math.sqrt(dim * (dim * dim - 1) / 12)
            sides.append(_unit(q) / norm if case["asymmetric"] else (_ranks(q) - (dim - 1) / 2).double() / norm / norm)
        else:
            norm = math.sqrt(dim * ((1 << bits) ** 2 - 1) / 12)
            sides.append(_centred(q, bits) / norm / norm if case.get("symmetric") else _unit(q) / norm)
        best.append(None)
    for _, docs in _corpus(case, seed, torch.empty_like(q)):
        for x in docs.split(32768):
            r = _ranks(x)
            for j, bits in enumerate(widths):
                d = r - (dim - 1) / 2 if op == "rank" else r * (1 << bits) // dim - ((1 << bits) - 1) / 2
                best[j] = _top(best[j], sides[j] @ d.double().T, k)
    if op != "mixed":
        return [best[0].flatten(), None]
    r = np.random.RandomState(seed & 0x7FFFFFFF)
    which = torch.from_numpy(r.randint(0, 3, case["nq"])).cuda()
    k_of = torch.tensor([10, 50, 100])[torch.from_numpy(r.randint(0, 3, case["nq"]))].cuda()
    k_of[0] = k
    rows = torch.stack(best)[which, torch.arange(case["nq"], device="cuda")]
    rows[torch.arange(rows.shape[1], device="cuda") >= k_of[:, None]] = -math.inf
    return [rows.flatten(), None]
