"""Exact rerank of batches whose queries name the same rows many times over: every transport fetches a row once, whether in one call, in
overlapped sub-batches or in a sharded session, batch after batch; rows no 16-byte load can take; candidates given twice."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def index(n, dim, u8, seed):
    rng = np.random.default_rng(seed)
    vec = rng.integers(0, 256, (n, dim)).astype(np.uint8) if u8 else rng.standard_normal((n, dim)).astype(np.float32)
    cen = rng.standard_normal((4, dim)).astype(np.float32)
    m = 4 if dim % 4 == 0 else 3
    return dict(centroids=cen, offsets=np.array([0, n // 4, n // 2, n // 2, n], np.int64), reordered_ids=rng.permutation(n).astype(np.int64),
                codes=rng.integers(0, 16, (n, m)).astype(np.uint8), codebook=rng.standard_normal((m, 16, dim // m)).astype(np.float32), vectors=vec)


@pytest.mark.parametrize("mode", [0, 1, 3, 4])
@pytest.mark.parametrize("dim,u8,nq,width", [(32, False, 700, 100), (33, False, 700, 100), (30, True, 70, 1000), (100, True, 700, 100), (9, True, 20, 64)])
def test_rows_named_many_times(psb, mode, dim, u8, nq, width):
    import torch
    ix = index(1500, dim, u8, dim + mode)
    rng = np.random.default_rng(nq)
    with psb.Session(ix, n_rerank=width, exact_mode=mode, max_batch=nq) as s:
        for again in range(3):
            q = rng.integers(0, 256, (nq, dim)).astype(np.uint8) if u8 else rng.standard_normal((nq, dim)).astype(np.float32)
            cand = np.stack([rng.permutation(1500)[:width] for _ in range(nq)]).astype(np.int32)
            cand[:, 5] = -1
            cand[::3, 7] = cand[::3, 3]          # a candidate twice
            cand[1, :] = cand[1, 0]              # only one row
            cnt = rng.integers(0, width + 1, nq).astype(np.int32)
            rows = torch.empty((nq, 10), dtype=torch.int32, device="cuda"); dist = torch.empty((nq, 10), device="cuda")
            s.stage_rerank(torch.from_numpy(q).cuda(), nq, torch.from_numpy(cand).cuda(), width, width, torch.from_numpy(cnt).cuda(), 10, rows, dist)
            s.sync()
            masked = np.where(np.arange(width)[None, :] < cnt[:, None], cand, -1)
            wi, wd = oracle.rerank(ix["vectors"], q, masked, 10)
            assert np.array_equal(rows.cpu().numpy(), wi) and np.array_equal(dist.cpu().numpy(), wd)


@pytest.mark.parametrize("scan_mode", [0, 3])
@pytest.mark.parametrize("mode", [0, 1, 4])
def test_overlapped_batches_share_rows(psb, mode, scan_mode):
    ix = index(3000, 32, False, 7)
    q = np.random.default_rng(8).standard_normal((2500, 32)).astype(np.float32)
    want = oracle.ivfpq_search(ix, q[:200], 3, 10, 60)
    with psb.Session(ix, n_rerank=60, exact_mode=3) as s:
        ref = s.search(q, 3, 10, batch_size=2500)
    with psb.Session(ix, n_rerank=60, exact_mode=mode, scan_mode=scan_mode) as s:
        for _ in range(2):
            got = s.search(q, 3, 10, batch_size=2500)
            assert np.array_equal(got["indices"], ref["indices"]) and np.array_equal(got["distances"], ref["distances"])
    assert np.array_equal(ref["indices"][:200], want["indices"]) and np.array_equal(ref["distances"][:200], want["distances"])


@pytest.mark.parametrize("dim,u8", [(16, False), (4, False), (20, False), (60, False), (64, False), (68, False), (112, False), (124, False), (128, False),
                                    (200, False), (960, False), (16, True), (128, True), (144, True), (272, True)])
@pytest.mark.parametrize("nq,width", [(2, 33), (90, 700)])
def test_rows_of_whole_units(psb, dim, u8, nq, width):
    import torch
    ix = index(900, dim, u8, dim)
    rng = np.random.default_rng(dim)
    with psb.Session(ix, n_rerank=width, exact_mode=3, max_batch=nq) as s:
        q = rng.integers(0, 256, (nq, dim)).astype(np.uint8) if u8 else rng.standard_normal((nq, dim)).astype(np.float32)
        cand = np.stack([rng.permutation(900)[:width] for _ in range(nq)]).astype(np.int32)
        cand[:, 5] = -1
        cnt = rng.integers(0, width + 1, nq).astype(np.int32)
        rows = torch.empty((nq, 10), dtype=torch.int32, device="cuda"); dist = torch.empty((nq, 10), device="cuda")
        s.stage_rerank(torch.from_numpy(q).cuda(), nq, torch.from_numpy(cand).cuda(), width, width, torch.from_numpy(cnt).cuda(), 10, rows, dist)
        s.sync()
        masked = np.where(np.arange(width)[None, :] < cnt[:, None], cand, -1)
        wi, wd = oracle.rerank(ix["vectors"], q, masked, 10)
        assert np.array_equal(rows.cpu().numpy(), wi) and np.array_equal(dist.cpu().numpy(), wd)


@pytest.mark.parametrize("how", ["alone", "share", "background"])
@pytest.mark.parametrize("dim,u8,nq,width", [(32, False, 507, 100), (32, False, 508, 100), (100, True, 700, 100), (33, False, 340, 100), (33, False, 700, 100)])
def test_hybrid_shares(psb, how, dim, u8, nq, width):
    """The hybrid transport by the kernel alone, with a share the caller names, and on a stream beside another: on both sides of the lines."""
    import torch
    ix = index(1500, dim, u8, dim)
    rng = np.random.default_rng(nq + dim)
    with psb.Session(ix, n_rerank=width, exact_mode=4, max_batch=nq, zero_copy_pct=40 if how == "share" else 0) as s:
        other = torch.cuda.Stream()
        if how == "background":
            s.set_stream(other.cuda_stream, background=True)
        for again in range(2):
            q = rng.integers(0, 256, (nq, dim)).astype(np.uint8) if u8 else rng.standard_normal((nq, dim)).astype(np.float32)
            cand = np.stack([rng.permutation(1500)[:width] for _ in range(nq)]).astype(np.int32)
            dq, dc = torch.from_numpy(q).cuda(), torch.from_numpy(cand).cuda()
            rows = torch.empty((nq, 10), dtype=torch.int32, device="cuda"); dist = torch.empty((nq, 10), device="cuda")
            torch.cuda.synchronize()
            s.stage_rerank(dq, nq, dc, width, width, None, 10, rows, dist)
            s.sync()
            torch.cuda.synchronize()
            wi, wd = oracle.rerank(ix["vectors"], q, cand, 10)
            assert np.array_equal(rows.cpu().numpy(), wi) and np.array_equal(dist.cpu().numpy(), wd)
        if how == "background":
            s.set_stream(None)


@pytest.mark.parametrize("count", [31, 32, 33, 32767, 32768, 32769, 70001])
@pytest.mark.parametrize("mode", [0, 4])
def test_slots_in_row_order(psb, mode, count):
    """Row counts at the ends of a word of marks and of a CTA's stretch of them, the first and last rows among those asked for, every row and few."""
    import torch
    ix = index(count, 32, False, count)
    rng = np.random.default_rng(count)
    nq, width = 900, 64                                             # above the line from which rows are fetched once
    with psb.Session(ix, n_rerank=width, exact_mode=mode, max_batch=nq) as s:
        for pool in (np.arange(count), np.unique(np.concatenate([[0, count - 1], rng.integers(0, count, 50)]))):
            q = rng.standard_normal((nq, 32)).astype(np.float32)
            cand = pool[rng.integers(0, len(pool), (nq, width))].astype(np.int32)
            cand[0, :2] = [0, count - 1]
            cand[:, 9] = -1
            rows = torch.empty((nq, 10), dtype=torch.int32, device="cuda"); dist = torch.empty((nq, 10), device="cuda")
            s.stage_rerank(torch.from_numpy(q).cuda(), nq, torch.from_numpy(cand).cuda(), width, width, None, 10, rows, dist)
            s.sync()
            wi, wd = oracle.rerank(ix["vectors"], q, cand, 10)
            assert np.array_equal(rows.cpu().numpy(), wi) and np.array_equal(dist.cpu().numpy(), wd)


@pytest.mark.parametrize("mode,pct", [(0, 0), (4, 0), (4, 60), (1, 0)])   # the kernel, without and with the option of host threads; with them; they alone
def test_cuts_of_a_large_batch(psb, mode, pct):
    """Batches large enough for uneven sub-batches, whatever the cuts: the results of one piece.  A number of sub-batches that the caller gives holds
    where the kernel fetches the rows: as many launches as of equal sub-batches."""
    ix = index(3000, 32, False, 9)
    q = np.random.default_rng(10).standard_normal((4201, 32)).astype(np.float32)
    with psb.Session(ix, n_rerank=60, exact_mode=3, serial_pipeline=True) as s:
        ref = s.search(q, 3, 10, batch_size=4201)

    def launches(**how):
        with psb.Session(ix, n_rerank=60, exact_mode=mode, zero_copy_pct=pct, **how) as s:
            for _ in range(2):
                got = s.search(q, 3, 10, batch_size=4201)
                assert np.array_equal(got["indices"], ref["indices"]) and np.array_equal(got["distances"], ref["distances"])
            return got["stats"]["kernel_launches"]
    own = [launches(even_cuts=e) for e in (0, 1, 2)]
    assert own[1] <= own[0] and own[1] == own[2]
    for parts in (2, 3, 4, 6):
        equal = launches(pipeline_parts=parts, even_cuts=1)
        assert mode not in (0, 4) or pct or launches(pipeline_parts=parts) == launches(pipeline_parts=parts, even_cuts=2) == equal
        assert parts <= 4 or launches(pipeline_parts=parts) == equal


@pytest.mark.parametrize("mode,pct", [(0, 0), (4, 0), (4, 50)])
def test_rows_fetched_are_counted(psb, mode, pct):
    """Each distinct row of a batch once, whoever brings it; rows that are scored in place are not counted."""
    import torch
    ix = index(1500, 32, False, 5)
    rng = np.random.default_rng(6)
    nq, width = 700, 100
    with psb.Session(ix, n_rerank=width, exact_mode=mode, zero_copy_pct=pct, max_batch=nq) as s:
        assert s.counters(reset=True)["rerank_rows_fetched"] == 0
        want = 0
        q = torch.from_numpy(rng.standard_normal((nq, 32)).astype(np.float32)).cuda()
        rows = torch.empty((nq, 10), dtype=torch.int32, device="cuda"); dist = torch.empty((nq, 10), device="cuda")
        for top in (300, 1500):
            cand = rng.integers(-1, top, (nq, width)).astype(np.int32)
            s.stage_rerank(q, nq, torch.from_numpy(cand).cuda(), width, width, None, 10, rows, dist)
            s.sync()
            want += len(np.unique(cand[cand >= 0]))
        s.stage_rerank(q, 3, torch.from_numpy(cand[:3].copy()).cuda(), width, width, None, 10, rows, dist)   # in place
        s.sync()
        assert s.counters(reset=True)["rerank_rows_fetched"] == want
        assert s.counters()["rerank_rows_fetched"] == 0


@pytest.mark.parametrize("mode,pct,call", [(0, 0, "search"), (4, 90, "search"), (4, 90, "stage")])   # the kernel alone; host threads beside it
def test_error_beside_a_gather(psb, mode, pct, call):
    """A call that ends with an error while a kernel on a stream of its own gathers its rows: the session's stream goes on behind the gather, so
    that the next call, or the owner of its buffers, does not meet it.  The transfer takes 7 ms; nothing is left of it once the stream has drained."""
    import time
    import torch
    n, dim, nq, width = 100000, 1024, 2100, 400
    ix = index(n, dim, False, 1)
    q = np.random.default_rng(2).standard_normal((nq, dim)).astype(np.float32)
    st = torch.cuda.Stream()
    with psb.Session(ix, n_rerank=width, exact_mode=mode, zero_copy_pct=pct, max_batch=nq, test_skip_mma=16, stream=st.cuda_stream) as s:
        dq = torch.from_numpy(q).cuda()
        ids, dist = torch.empty((nq, 10), dtype=torch.int64, device="cuda"), torch.empty((nq, 10), device="cuda")
        cand = torch.randint(n, (nq, width), dtype=torch.int32, device="cuda")
        rows = torch.empty((nq, 10), dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        for _ in range(2):
            with pytest.raises(psb.PsbError) as e:
                if call == "search":
                    s.search_device(dq, nq, 3, 10, ids, dist)
                else:
                    s.stage_rerank(dq, nq, cand, width, width, None, 10, rows, dist)
            assert e.value.status == 6 and "gather" in str(e.value)
            st.synchronize()
            t = time.perf_counter()
            torch.cuda.synchronize()
            assert time.perf_counter() - t < 2.5e-3
    with psb.Session(ix, n_rerank=width, exact_mode=mode, zero_copy_pct=pct, max_batch=nq) as s:   # the rows are mapped anew
        got = s.search(q, 3, 10, batch_size=nq)
    want = oracle.ivfpq_search(ix, q[-8:], 3, 10, width)
    assert np.array_equal(got["indices"][-8:], want["indices"]) and np.array_equal(got["distances"][-8:], want["distances"])
