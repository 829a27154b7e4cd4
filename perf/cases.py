"""Workloads the library's speed is judged by, each through the entry points a user's program calls.

An index is a Gaussian mixture with one inverted list per component, as in the repository's benchmark configurations; sizes are
those configurations cut down so that inputs are made in a fraction of a second.  A case is a dict of plain values:

  search     IVF-PQ search: a session over an index, host arrays in and out or device tensors in and out
  flat       IVF-Flat search over device-resident rows
  coarse     the coarse stage alone: the nearest centroids of each query
  kmeans     Lloyd iterations on device rows
  pq_train   PQ codebooks on device rows
  pq_encode  PQ codes of device rows
  sign       candidate search of the 1-bit sign codec, host queries and probes in, candidate rows out
"""
import math

import numpy as np
import torch

from paraselect_b200 import api

K = 256  # codewords per sub-quantiser: 8-bit codes


def listed():
    return [
        # online serving: one query per call, rows for the exact rerank in host memory; latency and launches count
        dict(name="search_one", kind="search", adc="plain", rows="fp32", place="mapped", io="host", n=1_000_000, dim=96, M=48,
             nlist=1024, zipf=0.0, sigma=0.25, nq=1, nprobe=32, k=10, rerank=100),
        # byte vectors of a dimension that is no multiple of 8, five elements per code, an odd batch and list count
        dict(name="search_odd_u8", kind="search", adc="plain", rows="u8", place="mapped", io="host", n=500_000, dim=100, M=20,
             nlist=701, zipf=0.0, sigma=0.25, nq=333, nprobe=20, k=10, rerank=200),
        # the benchmark's 1M x 128 configuration as it is: a large batch, host in and out, rows mapped
        dict(name="search_batch", kind="search", adc="plain", rows="fp32", place="mapped", io="host", n=1_000_000, dim=128, M=32,
             nlist=1024, zipf=0.0, sigma=0.25, nq=10_000, nprobe=32, k=10, rerank=100),
        # the benchmark's large configuration cut down: skewed lists, wide candidate lists, both host transports at once
        dict(name="search_skewed", kind="search", adc="plain", rows="fp32", place="hybrid", io="device", n=2_000_000, dim=96, M=48,
             nlist=4096, zipf=1.1, sigma=0.25, nq=4096, nprobe=64, k=100, rerank=1000),
        # residual codes, rows for the rerank already on the GPU: the scan and the selection are all there is
        dict(name="search_residual", kind="search", adc="residual", rows="fp32", place="resident", io="device", n=2_000_000, dim=96,
             M=48, nlist=2048, zipf=0.0, sigma=0.25, nq=2000, nprobe=32, k=10, rerank=500),
        # a handful of exact searches from a service
        dict(name="flat_few", kind="flat", io="host", n=300_000, dim=96, nlist=512, sigma=0.3, nq=4, nprobe=32, k=20),
        # the benchmark's IVF-Flat configuration
        dict(name="flat_batch", kind="flat", io="device", n=100_000, dim=128, nlist=256, sigma=0.3, nq=1000, nprobe=16, k=10),
        # the benchmark's coarse-only configuration, a fifth of its queries
        dict(name="coarse_wide", kind="coarse", nlist=65_536, dim=96, nq=20_000, k=64),
        # index build: coarse centroids
        dict(name="kmeans", kind="kmeans", n=400_000, dim=128, components=4096, sigma=0.3, k=8192, iters=5),
        # index build: codebooks on a training sample of 128 rows per codeword
        dict(name="pq_train", kind="pq_train", n=32_768, dim=96, M=24, iters=10),
        # index build: the codes of all rows
        dict(name="pq_encode", kind="pq_encode", n=1_000_000, dim=128, M=32),
        # the benchmark's sign-codec configuration, a tenth of its rows
        dict(name="sign_search", kind="sign", mode="float", n=2_000_000, dim=128, nlist=2048, nq=4000, nprobe=32, k=512),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["search", "search", "search", "flat", "flat", "coarse", "kmeans", "pq_train", "pq_encode", "sign"])
    if kind == "search":
        dim, m = rng.choice([(32, 8), (64, 16), (96, 24), (96, 48), (100, 20), (128, 16), (128, 32), (128, 64)])
        c = dict(kind=kind, adc=rng.choice(["plain", "plain", "residual"]), rows=rng.choice(["fp32", "fp32", "u8"]),
                 place=rng.choice(["mapped", "resident", "hybrid"]), io=rng.choice(["host", "device"]), n=_log(rng, 100_000, 2_000_000),
                 dim=dim, M=m, nlist=_log(rng, 256, 4096), zipf=rng.choice([0.0, 0.0, 1.1]), sigma=0.25, nq=_log(rng, 1, 10_000),
                 nprobe=_log(rng, 4, 64), k=_log(rng, 1, 100))
        c["rerank"] = min(1000, c["k"] * _log(rng, 4, 20))
        if c["adc"] == "residual" and dim == 100:  # a table per (query, probe): small batches
            c["nq"] = 1 + c["nq"] % 500
        width = max(c["rerank"], 512) if c["adc"] == "residual" else c["rerank"]
        host_bytes = width * dim * (4 if c["rows"] == "fp32" else 1) * (1 if c["place"] != "resident" else 0.02)
        c["nq"] = max(1, min(c["nq"], int(1.5e9 / host_bytes), int(6e8 / (c["nprobe"] * c["n"] / c["nlist"] + 0.05 * c["zipf"] * c["n"]))))
        return c
    if kind == "flat":
        c = dict(kind=kind, io=rng.choice(["host", "device"]), n=_log(rng, 20_000, 300_000), dim=rng.choice([32, 64, 96, 100, 126, 128]),
                 nlist=_log(rng, 64, 512), sigma=0.3, nq=_log(rng, 1, 1000), nprobe=_log(rng, 4, 32), k=_log(rng, 1, 100))
        c["nq"] = max(1, min(c["nq"], int(8e8 * c["nlist"] / (c["nprobe"] * c["n"] * c["dim"]))))
        return c
    if kind == "coarse":
        return dict(kind=kind, nlist=_log(rng, 1024, 65_536), dim=rng.choice([64, 96, 100, 120]), nq=_log(rng, 1, 20_000), k=_log(rng, 1, 64))
    if kind == "kmeans":
        return dict(kind=kind, n=_log(rng, 20_000, 400_000), dim=rng.choice([64, 96, 100, 128]), components=_log(rng, 100, 4096),
                    sigma=0.3, k=_log(rng, 64, 8192), iters=rng.randint(2, 5))
    if kind in ("pq_train", "pq_encode"):
        dim, m = rng.choice([(64, 16), (96, 24), (96, 48), (100, 20), (128, 16), (128, 32)])
        if kind == "pq_encode":
            return dict(kind=kind, n=_log(rng, 1000, 1_000_000), dim=dim, M=m)
        n = _log(rng, 4096, 400_000)
        if n <= 78_125:  # samples this small are seeded by k-means++: no more work than the listed case
            n = min(n, 32_768 * 24 // m)
        return dict(kind=kind, n=n, dim=dim, M=m, iters=rng.randint(4, 10))
    return dict(kind=kind, mode=rng.choice(["float", "float", "coded"]), n=_log(rng, 100_000, 2_000_000), dim=rng.choice([64, 96, 100, 128]),
                nlist=_log(rng, 256, 2048), nq=_log(rng, 1, 4000), nprobe=_log(rng, 4, 32), k=_log(rng, 64, 512))


# ---- inputs -----------------------------------------------------------------------------------------------------------

_stream = None


def stream():
    """The stream of the user's program: sessions and operators are given it."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


def mixture(gen, n, dim, ncomp, sigma, zipf=0.0):
    """Centres, rows in component order, row offsets of the components, weights of the components."""
    w = 1.0 / np.arange(1, ncomp + 1) ** zipf
    w /= w.sum()
    offsets = np.floor(np.concatenate([[0.0], np.cumsum(w)]) * n + 1e-6).astype(np.int64)
    offsets[-1] = n
    centres = torch.randn(ncomp, dim, device="cuda", generator=gen)
    rows = torch.randn(n, dim, device="cuda", generator=gen).mul_(sigma)
    rows += torch.repeat_interleave(centres, torch.from_numpy(np.diff(offsets)).cuda(), dim=0, output_size=n)
    return centres, rows, offsets, w


def queries_near(gen, centres, w, nq, sigma):
    comp = torch.multinomial(torch.from_numpy(w).cuda(), nq, replacement=True, generator=gen)
    return centres[comp] + sigma * torch.randn(nq, centres.shape[1], device="cuda", generator=gen)


def bytes_of(x):
    """The same values as byte vectors have them: whole numbers from 0 to 255."""
    return (x * 40 + 128).round_().clamp_(0, 255)


def codebooks(gen, rows, m, iters=3, sample=8192):
    """[m][K][dim / m] codewords: a few Lloyd iterations on a sample, the same for every caller."""
    take = torch.randperm(rows.shape[0], device="cuda", generator=gen)[:sample]
    x = rows[take].view(take.numel(), m, -1).transpose(0, 1).contiguous()
    c = x[:, :K].clone()
    for _ in range(iters):
        near = torch.baddbmm(c.square().sum(2)[:, None, :], x, c.transpose(1, 2), alpha=-2.0).argmin(2, keepdim=True)
        one = torch.zeros(m, x.shape[1], K, device="cuda").scatter_(2, near, 1.0)
        count = one.sum(1)[:, :, None]
        c = torch.where(count > 0, torch.bmm(one.transpose(1, 2), x) / count.clamp(min=1.0), c)
    return c.contiguous()


def host(x):
    return x.cpu().numpy()


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    return globals()["prepare_" + case["kind"]](case, gen)


def prepare_search(c, gen):
    n, dim, m, nq, k = c["n"], c["dim"], c["M"], c["nq"], c["k"]
    centres, rows, offsets, w = mixture(gen, n, dim, c["nlist"], c["sigma"], c["zipf"])
    q = queries_near(gen, centres, w, nq, c["sigma"])
    if c["rows"] == "u8":
        centres, rows, q = centres * 40 + 128, bytes_of(rows), bytes_of(q)
    coded = rows
    if c["adc"] == "residual":
        coded = rows - torch.repeat_interleave(centres, torch.from_numpy(np.diff(offsets)).cuda(), dim=0, output_size=n)
    book = codebooks(gen, coded, m)
    codes = torch.empty(n, m, dtype=torch.uint8, device="cuda")
    api.pq_encode(coded, n, dim, book, m, K, codes)
    ids = torch.randperm(n, device="cuda", generator=gen)
    u8 = rows.to(torch.uint8) if c["rows"] == "u8" else None
    vectors = rows if u8 is None else u8
    index = dict(centroids=host(centres), offsets=offsets, reordered_ids=host(ids), codes=host(codes), codebook=host(book),
                 vectors=vectors if c["place"] == "resident" else host(vectors))
    mode = dict(mapped=api.EXACT_HOST_MAPPED, resident=api.EXACT_RESIDENT, hybrid=api.EXACT_HOST_HYBRID)[c["place"]]
    session = api.Session(index, n_rerank=c["rerank"], exact_mode=mode, max_batch=nq, residual=c["adc"] == "residual",
                          stream=stream().cuda_stream)
    q_u8 = q.to(torch.uint8) if u8 is not None else None
    if c["io"] == "host":
        return dict(case=c, session=session, q=host(q), q_u8=host(q_u8) if q_u8 is not None else None)
    return dict(case=c, session=session, q=q, q_u8=q_u8, ids=torch.empty(nq, k, dtype=torch.int64, device="cuda"),
                dist=torch.empty(nq, k, device="cuda"))


def prepare_flat(c, gen):
    centres, rows, offsets, w = mixture(gen, c["n"], c["dim"], c["nlist"], c["sigma"])
    q = queries_near(gen, centres, w, c["nq"], c["sigma"])
    index = dict(centroids=host(centres), offsets=offsets, reordered_ids=host(torch.randperm(c["n"], device="cuda", generator=gen)),
                 vectors=host(rows))
    session = api.FlatSession(index, max_batch=c["nq"], stream=stream().cuda_stream)
    if c["io"] == "host":
        return dict(case=c, session=session, q=host(q))
    return dict(case=c, session=session, q=q, ids=torch.empty(c["nq"], c["k"], dtype=torch.int64, device="cuda"),
                dist=torch.empty(c["nq"], c["k"], device="cuda"))


def prepare_coarse(c, gen):
    nlist, dim = c["nlist"], c["dim"]
    cen = torch.randn(nlist, dim, device="cuda", generator=gen)
    q = torch.randn(c["nq"], dim, device="cuda", generator=gen)
    cen /= cen.norm(dim=1).mean()
    q /= q.norm(dim=1).mean()
    # the stage belongs to a session: an index of one row per list carries it
    index = dict(centroids=host(cen), offsets=np.arange(nlist + 1, dtype=np.int64), reordered_ids=np.arange(nlist, dtype=np.int64),
                 codes=np.zeros((nlist, 4), np.uint8), codebook=np.zeros((4, K, dim // 4), np.float32))
    session = api.Session(index, max_batch=c["nq"], stream=stream().cuda_stream)
    return dict(case=c, session=session, q=q, ids=torch.empty(c["nq"], c["k"], dtype=torch.int32, device="cuda"),
                dist=torch.empty(c["nq"], c["k"], device="cuda"))


def prepare_kmeans(c, gen):
    _, rows, _, _ = mixture(gen, c["n"], c["dim"], c["components"], c["sigma"])
    rows = rows[torch.randperm(c["n"], device="cuda", generator=gen)].contiguous()
    return dict(case=c, rows=rows, init=rows[: c["k"]].clone(), cen=torch.empty(c["k"], c["dim"], device="cuda"),
                assign=torch.empty(c["n"], dtype=torch.int32, device="cuda"))


def prepare_pq_train(c, gen):
    # residuals of rows against their centroids: what a residual index trains on, with the spread of each dimension its own
    rows = torch.randn(c["n"], c["dim"], device="cuda", generator=gen) * (0.1 + torch.rand(c["dim"], device="cuda", generator=gen))
    return dict(case=c, rows=rows, book=torch.empty(c["M"], K, c["dim"] // c["M"], device="cuda"))


def prepare_pq_encode(c, gen):
    s = prepare_pq_train(c, gen)
    x = s["rows"] if c["n"] >= 1024 else torch.randn(1024, c["dim"], device="cuda", generator=gen)
    return dict(case=c, rows=s["rows"], book=codebooks(gen, x, c["M"]),
                codes=torch.empty(c["n"], c["M"], dtype=torch.uint8, device="cuda"))


def prepare_sign(c, gen):
    centres, rows, offsets, w = mixture(gen, c["n"], c["dim"], c["nlist"], 0.25)
    q = queries_near(gen, centres, w, c["nq"], 0.25)
    near = torch.cdist(q, centres).topk(c["nprobe"], dim=1, largest=False).indices
    index = api.SignIndex()
    index.build_u8(host(bytes_of(rows).to(torch.uint8)), host(centres * 40 + 128), offsets)
    return dict(case=c, index=index, q=host(q * 40 + 128), probes=host(near.to(torch.int32)))


# ---- one pass ---------------------------------------------------------------------------------------------------------


def run(s):
    c = s["case"]
    kind = c["kind"]
    st = stream().cuda_stream
    if kind == "search":
        if c["io"] == "host":
            r = s["session"].search(s["q"], c["nprobe"], c["k"], queries_u8=s["q_u8"])
            return dict(ids=r["indices"], dist=r["distances"])
        s["session"].search_device(s["q"], c["nq"], c["nprobe"], c["k"], s["ids"], s["dist"], d_queries_u8=s["q_u8"])
        return dict(ids=s["ids"], dist=s["dist"])
    if kind == "flat":
        if c["io"] == "host":
            r = s["session"].search(s["q"], c["nprobe"], c["k"])
            return dict(ids=r["indices"], dist=r["distances"])
        s["session"].search_device(s["q"], c["nq"], c["nprobe"], c["k"], s["ids"], s["dist"])
        return dict(ids=s["ids"], dist=s["dist"])
    if kind == "coarse":
        s["session"].stage_coarse(s["q"], c["nq"], c["k"], s["ids"], s["dist"])
        return dict(ids=s["ids"], dist=s["dist"])
    if kind == "kmeans":
        with torch.cuda.stream(stream()):
            s["cen"].copy_(s["init"])
        objective = api.kmeans_train(s["rows"], c["n"], c["dim"], s["cen"], c["k"], c["iters"], s["assign"], stream=st)
        return dict(centroids=s["cen"], assign=s["assign"], objective=objective)
    if kind == "pq_train":
        api.pq_train(s["rows"], c["n"], c["dim"], c["M"], K, c["iters"], 42, s["book"], stream=st)
        return s["book"]
    if kind == "pq_encode":
        api.pq_encode(s["rows"], c["n"], c["dim"], s["book"], c["M"], K, s["codes"], stream=st)
        return s["codes"]
    mode = api.SIGN_FLOAT_STATES if c["mode"] == "float" else api.SIGN_CODED_STATES
    return s["index"].search_candidates(s["q"], s["probes"], c["k"], score_mode=mode)


# ---- what a pass cannot do without ------------------------------------------------------------------------------------


def scanned(c):
    """Expected rows one query scans, and rows the whole batch reads at least once."""
    w = 1.0 / np.arange(1, c["nlist"] + 1) ** c.get("zipf", 0.0)
    w /= w.sum()
    per = c["n"] * (float((w * w).sum()) + (c["nprobe"] - 1) / c["nlist"])
    seen = c["n"] * float((w * (1 - (1 - w) ** c["nq"] * (1 - 1 / c["nlist"]) ** (c["nq"] * (c["nprobe"] - 1)))).sum())
    return min(per, c["n"]), min(seen, c["n"])


def work(case):
    c = case
    kind, dim = c["kind"], c["dim"]
    if kind in ("search", "flat", "sign"):
        per, seen = scanned(c)
        coarse = c["nlist"] * dim * 4 + c["nq"] * dim * 4
        if kind == "flat":
            return dict(bytes=coarse + seen * dim * 4 + c["nq"] * c["k"] * 12, flops=2.0 * c["nq"] * dim * (c["nlist"] + 1.5 * per))
        if kind == "sign":
            return dict(bytes=coarse + c["nq"] * c["nprobe"] * 4 + seen * (dim / 8 + 4) + c["nq"] * c["k"] * 4, flops=1.0 * c["nq"] * per * dim)
        elem = 4 if c["rows"] == "fp32" else 1
        width = max(c["rerank"], c["k"], 512) if c["adc"] == "residual" else max(c["rerank"], c["k"])
        exact = c["nq"] * min(width, per) * dim if c["adc"] == "residual" or c["rerank"] > c["k"] else 0
        return dict(bytes=coarse + seen * c["M"] + exact * elem + c["nq"] * c["k"] * 12,
                    flops=2.0 * c["nq"] * dim * c["nlist"] + 3.0 * c["nq"] * K * dim + 1.0 * c["nq"] * per * c["M"] + 3.0 * exact)
    if kind == "coarse":
        return dict(bytes=(c["nlist"] + c["nq"]) * dim * 4 + c["nq"] * c["k"] * 8, flops=2.0 * c["nq"] * c["nlist"] * dim)
    if kind == "kmeans":
        passes = c["iters"] + 1
        return dict(bytes=passes * (c["n"] * dim * 4 + c["k"] * dim * 4) + c["n"] * 4, flops=2.0 * passes * c["n"] * c["k"] * dim)
    if kind == "pq_train":
        return dict(bytes=c["n"] * dim * 4 * c["iters"] + K * dim * 4, flops=2.0 * c["n"] * K * dim * (c["iters"] + 1))
    return dict(bytes=c["n"] * (dim * 4 + c["M"]) + K * dim * 4, flops=3.0 * c["n"] * K * dim)


def tolerance(case):
    """Searches and encodings are the same bits whatever computes them.  Training sums in 64 bits and rounds once, but a row that lies
    within rounding of two centroids may go to either, and moves its centroid by its share."""
    if case["kind"] == "kmeans":
        return dict(rel=1e-5, max=0.02, differ=1e-4)
    if case["kind"] == "pq_train":
        return dict(rel=1e-4, max=0.05)
    return "exact"
