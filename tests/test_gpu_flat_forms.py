"""IVF-Flat: the list form (many visitors per list) and the row form (few), tiles and row blocks that do not fill, dimensions that are no
multiple of four, and every way the selection can go - all values gathered, cut by the group minima, radix passes for equal values and
for more results than the minima cover - against the CPU checker."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dim,nlist,nq,nprobe,topk,values", [
    (3000, 33, 5, 97, 5, 10, "normal"), (3000, 100, 5, 1, 3, 7, "normal"), (4000, 64, 3, 33, 2, 300, "normal"), (9000, 16, 7, 2, 7, 300, "normal"),
    (6000, 8, 4, 40, 4, 1100, "normal"), (6000, 8, 4, 3, 4, 2048, "normal"), (7000, 12, 3, 40, 3, 50, "grid"), (5000, 4, 2, 2, 2, 20, "equal"),
    (64, 300, 2, 20, 2, 5, "normal"), (40, 7, 20, 33, 20, 64, "normal"), (30000, 2, 4, 200, 4, 300, "grid"), (30000, 1, 4, 3, 4, 900, "grid")])
def test_flat_forms(psb, n, dim, nlist, nq, nprobe, topk, values):
    rng = np.random.default_rng(n + dim + nq)
    draw = {"normal": lambda *s: rng.standard_normal(s), "grid": lambda *s: rng.integers(-1, 2, s), "equal": lambda *s: np.ones(s)}[values]
    cuts = np.sort(rng.integers(0, n + 1, nlist - 1))
    off = np.concatenate([[0], cuts, [n]]).astype(np.int64)
    fx = dict(centroids=rng.standard_normal((nlist, dim)).astype(np.float32), offsets=off, reordered_ids=rng.permutation(n).astype(np.int64),
              vectors=draw(n, dim).astype(np.float32))
    q = draw(nq, dim).astype(np.float32)
    wi, wd = oracle.ivfflat_search(fx["centroids"], off, fx["reordered_ids"], fx["vectors"], q, nprobe, topk)
    with psb.FlatSession(fx) as s:
        got = s.search(q, nprobe, topk)
    assert np.array_equal(got["indices"], wi) and np.array_equal(got["distances"], wd)


@pytest.mark.parametrize("nq,nlist,dim,k", [(1, 3, 5, 3), (33, 65, 12, 20), (2, 3000, 40, 1), (3, 5000, 8, 700), (40, 513, 6, 130), (2, 9000, 4, 1500),
                                           (30, 600, 5, 256), (30, 513, 5, 228), (30, 2000, 5, 900), (30, 2000, 5, 400), (3, 4000, 5, 512), (30, 1024, 5, 900)])   # the bound with few values for each wanted
@pytest.mark.parametrize("equal", [False, True])
def test_coarse_small_batches(psb, nq, nlist, dim, k, equal):
    rng = np.random.default_rng(nlist)
    c = rng.standard_normal((nlist, dim)).astype(np.float32)
    if equal:
        c[:] = c[0]
    q = rng.standard_normal((nq, dim)).astype(np.float32)
    ids, dist = psb.coarse_host(q, c, k, coarse_mode=1)
    wi, wd = oracle.coarse(q, c, k)
    assert np.array_equal(ids, wi) and np.array_equal(dist, wd)


@pytest.mark.parametrize("n,dim,nlist,nq,nprobe,topk,values", [
    # enough to visit (4e7 dimensions, two visitors a list) for the list form
    (3000, 33, 5, 700, 5, 10, "normal"), (3000, 100, 5, 251, 4, 7, "normal"), (4000, 64, 3, 385, 2, 300, "normal"), (9000, 16, 7, 449, 7, 300, "normal"),
    (6000, 8, 4, 1300, 4, 1100, "normal"), (6000, 8, 4, 1251, 4, 2048, "normal"), (7000, 12, 3, 750, 3, 50, "grid"), (5000, 4, 2, 3200, 2, 20, "equal"),
    (64, 300, 2, 3300, 2, 5, "normal"), (400, 7, 20, 22000, 20, 64, "normal"), (30000, 2, 4, 1100, 4, 300, "grid"), (30000, 1, 4, 2100, 4, 900, "grid"),
    # more queries than one part of a call holds, in the row form and in the list form; more than 2^28 distances
    (40, 7, 20, 33000, 20, 64, "normal"), (300, 16, 4, 33001, 4, 10, "normal"), (600001, 2, 3, 500, 3, 10, "normal")])
def test_flat_list_form_and_parts(psb, n, dim, nlist, nq, nprobe, topk, values):
    rng = np.random.default_rng(n + dim + nq)
    draw = {"normal": lambda *s: rng.standard_normal(s), "grid": lambda *s: rng.integers(-1, 2, s), "equal": lambda *s: np.ones(s)}[values]
    off = np.concatenate([[0], np.sort(rng.integers(0, n + 1, nlist - 1)), [n]]).astype(np.int64)
    fx = dict(centroids=rng.standard_normal((nlist, dim)).astype(np.float32), offsets=off, reordered_ids=rng.permutation(n).astype(np.int64),
              vectors=draw(n, dim).astype(np.float32))
    q = draw(nq, dim).astype(np.float32)
    with psb.FlatSession(fx, max_batch=nq) as s:
        got = s.search(q, nprobe, topk, batch_size=nq)
    some = np.unique(np.concatenate([np.arange(50), nq // 2 + np.arange(-25, 25), nq - 1 - np.arange(50), rng.integers(0, nq, 100)]))   # part borders among them
    wi, wd = oracle.ivfflat_search(fx["centroids"], off, fx["reordered_ids"], fx["vectors"], q[some], nprobe, topk)
    assert np.array_equal(got["indices"][some], wi) and np.array_equal(got["distances"][some], wd)


@pytest.mark.parametrize("dim", [5, 16, 100, 128, 130, 240, 256])
@pytest.mark.parametrize("kind", ["normal", "far", "tiny", "vanish", "grid", "odd", "one", "spread", "crowd", "large"])
@pytest.mark.parametrize("k", [1, 10, 256])
def test_list_form_behind_the_filter(psb, dim, kind, k):
    """Approximate distances and exact evaluation of the candidates: a large offset, which loosens the bound; values whose squares vanish, and
    ones whose products with the query lie on both sides of the smallest normal number; equal distances by the hundred and values that are not finite; a row and rows of many times the others' norm; a list of equal rows, whose visitors
    alone go back to the exact tiles; norms on both sides of the largest that a bound is given for."""
    rng = np.random.default_rng(dim + k)
    nlist, n, nq, nprobe = 6, 9000, 700, 3
    cen = rng.standard_normal((nlist, dim)).astype(np.float32)
    off = np.array([0, 1, 65, 65, 1400, 5000, n], np.int64)
    own = np.repeat(np.arange(nlist), np.diff(off))
    x = (cen[own] + 0.3 * rng.standard_normal((n, dim))).astype(np.float32)
    q = (cen[rng.integers(0, nlist, nq)] + 0.3 * rng.standard_normal((nq, dim))).astype(np.float32)
    if kind == "far":
        x, q, cen = x + 100, q + 100, cen + 100
    if kind == "tiny":
        x, q, cen = (v * np.float32(1e-20) for v in (x, q, cen))
    if kind == "vanish":
        x, cen, q = x * np.float32(1e-17), cen * np.float32(1e-17), q * np.float32(1e-21)
    if kind == "grid":
        x, q = np.round(x), np.round(q)
    if kind == "one":
        x[2000] *= 1000
    if kind == "spread":
        x[::3] *= np.exp(rng.uniform(-7, 7, (len(x[::3]), 1))).astype(np.float32)
    if kind == "crowd":
        x[1400:5000] = cen[4]
    if kind == "large":
        x, q, cen = (v * np.float32(4e17 / np.sqrt(dim)) for v in (x, q, cen))
        x[::2] *= 3
    if kind == "odd":
        x[4000, 0], x[77, dim - 1], q[3, 1] = np.inf, np.nan, np.inf
    ix = dict(centroids=cen, offsets=off, reordered_ids=rng.permutation(n).astype(np.int64), vectors=x)
    with psb.FlatSession(ix, max_batch=nq, scan_mode=3) as s:
        got = s.search(q, nprobe, k, batch_size=nq, want_coarse=True)
    for i in list(range(12)) + [nq - 1]:
        rows = np.concatenate([np.arange(off[p], off[p + 1]) for p in got["coarse"][i]])
        d = np.zeros(len(rows), np.float32)
        with np.errstate(invalid="ignore", over="ignore"):
            for j in range(dim):
                t = q[i, j] - x[rows, j]
                d += t * t
        fine = np.isfinite(d)
        if not fine.all() and i == 3:
            continue
        order = np.lexsort((rows, np.where(np.isnan(d), np.inf, d)))[:k]
        take = np.isfinite(d[order])
        assert np.array_equal(got["indices"][i][: len(order)][take], ix["reordered_ids"][rows[order]][take]), (kind, i)
        assert np.array_equal(got["distances"][i][: len(order)][take], d[order][take])


@pytest.mark.parametrize("form", [0, 1, 3])
@pytest.mark.parametrize("nprobe,k", [(1, 10), (1, 11), (1, 256), (2, 200), (3, 256), (3, 200)])   # either side of the line: rows, and rows for each wanted
def test_both_forms_of_the_tiles(psb, form, nprobe, k):
    rng = np.random.default_rng(k)
    n, dim, nlist, nq = 9300, 64, 7, 1100
    off = np.linspace(0, n, nlist + 1).astype(np.int64)
    fx = dict(centroids=rng.standard_normal((nlist, dim)).astype(np.float32), offsets=off, reordered_ids=rng.permutation(n).astype(np.int64),
              vectors=rng.standard_normal((n, dim)).astype(np.float32))
    q = rng.standard_normal((nq, dim)).astype(np.float32)
    with psb.FlatSession(fx, max_batch=nq, scan_mode=form) as s:
        got = s.search(q, nprobe, k, batch_size=nq)
    some = rng.integers(0, nq, 60)
    wi, wd = oracle.ivfflat_search(fx["centroids"], off, fx["reordered_ids"], fx["vectors"], q[some], nprobe, k)
    assert np.array_equal(got["indices"][some], wi) and np.array_equal(got["distances"][some], wd)


def test_calls_of_changing_size(psb):
    """A session's buffers are one allocation, laid out anew when a call needs more: both forms, more and fewer queries, probes and results."""
    rng = np.random.default_rng(3)
    n, dim, nlist = 20000, 64, 32
    off = np.concatenate([[0], np.sort(rng.integers(0, n + 1, nlist - 1)), [n]]).astype(np.int64)
    fx = dict(centroids=rng.standard_normal((nlist, dim)).astype(np.float32), offsets=off, reordered_ids=rng.permutation(n).astype(np.int64),
              vectors=rng.standard_normal((n, dim)).astype(np.float32))
    with psb.FlatSession(fx, max_batch=900) as s:
        for nq, nprobe, topk in ((3, 8, 10), (700, 4, 10), (5, 32, 300), (900, 2, 256), (64, 20, 7), (900, 9, 300), (1, 1, 1), (850, 3, 20)):
            q = rng.standard_normal((nq, dim)).astype(np.float32)
            got = s.search(q, nprobe, topk, batch_size=nq)
            wi, wd = oracle.ivfflat_search(fx["centroids"], off, fx["reordered_ids"], fx["vectors"], q, nprobe, topk)
            assert np.array_equal(got["indices"], wi) and np.array_equal(got["distances"], wd)


@pytest.mark.parametrize("kind,times", [("one", 2.0), ("nan", 2.0), ("far", 4.0), ("same", 6.0)])   # measured 1.0, 1.0, 2.3, 3.7
def test_cost_where_the_bound_is_loose(psb, kind, times):
    """Rows that loosen the filter's bound cost the queries that it cannot serve the exact tiles, and the others nothing."""
    import torch
    rng = np.random.default_rng(1)
    n, dim, nlist, nq = 100000, 128, 256, 1000
    cen = rng.standard_normal((nlist, dim)).astype(np.float32)
    own = np.sort(rng.integers(0, nlist, n))
    off = np.concatenate([[0], np.cumsum(np.bincount(own, minlength=nlist))]).astype(np.int64)
    x = (cen[own] + 0.3 * rng.standard_normal((n, dim))).astype(np.float32)
    q = (cen[rng.integers(0, nlist, nq)] + 0.3 * rng.standard_normal((nq, dim))).astype(np.float32)

    def cost(x, q, cen):
        st = torch.cuda.Stream()
        with psb.FlatSession(dict(centroids=cen, offsets=off, reordered_ids=np.arange(n), vectors=x), max_batch=nq, stream=st.cuda_stream) as s:
            dq, ids, dist = torch.from_numpy(q).cuda(), torch.empty(nq, 10, dtype=torch.int64, device="cuda"), torch.empty(nq, 10, device="cuda")
            torch.cuda.synchronize()
            ms = []
            for _ in range(9):
                a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                a.record(st)
                for _ in range(4):
                    s.search_device(dq, nq, 16, 10, ids, dist)
                b.record(st)
                torch.cuda.synchronize()
                ms.append(a.elapsed_time(b))
        return min(ms)   # the host's other work only adds
    plain = cost(x, q, cen)
    if kind == "one":
        x[n // 2] *= 1000
    if kind == "nan":
        x[n // 2, 0] = np.nan
    if kind == "far":
        x, q, cen = x + 100, q + 100, cen + 100
    if kind == "same":
        x[:] = 1.0
    assert cost(x, q, cen) < times * plain
