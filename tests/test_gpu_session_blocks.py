"""Sessions hand their page-locked block on: many at once, in threads, one after the other, on other streams, with calls that pass their
queries and results through the block and calls too large for it."""
import threading

import numpy as np
import pytest

import oracle
import synth

pytestmark = pytest.mark.gpu


def test_blocks_pass_between_sessions(psb):
    ix = synth.make_index(4000, 32, 16, 8, seed=5)
    q = synth.make_queries(ix, 3000, seed=6)
    want = oracle.ivfpq_search(ix, q, 4, 10, 40)
    fx = dict(centroids=ix["centroids"], offsets=ix["offsets"], reordered_ids=ix["reordered_ids"], vectors=ix["vectors"])
    fi, fd = oracle.ivfflat_search(fx["centroids"], fx["offsets"], fx["reordered_ids"], fx["vectors"], q, 4, 10)
    wrong = []

    def check(s, lo, n, flat):
        got = s.search(q[lo:lo + n], 4, 10)
        wi, wd = (fi, fd) if flat else (want["indices"], want["distances"])
        if not (np.array_equal(got["indices"], wi[lo:lo + n]) and np.array_equal(got["distances"], wd[lo:lo + n])):
            wrong.append((lo, n, flat))

    def work(t):
        try:
            rng = np.random.default_rng(t)
            for i in range(6):
                flat = (t + i) % 3 == 0
                with (psb.FlatSession(fx, max_batch=3000) if flat else psb.Session(ix, n_rerank=40, max_batch=3000)) as s:
                    for n in (1, 300, 3000 if i == 2 else 7, 1):
                        check(s, int(rng.integers(0, 3001 - n)), n, flat)
        except Exception as e:  # noqa: BLE001 - reported by the test below
            wrong.append(repr(e))

    threads = [threading.Thread(target=work, args=(t,)) for t in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong
    held = [psb.Session(ix, n_rerank=40, max_batch=64) for _ in range(12)]   # more than are kept between sessions
    for i, s in enumerate(held):
        check(s, i * 50, 50, False)
    for s in held:
        s.close()
    with psb.Session(ix, n_rerank=40, max_batch=64) as s:
        check(s, 0, 64, False)
    assert not wrong, wrong


@pytest.mark.parametrize("mode", [0, 1, 4])       # mapped, staged, hybrid
@pytest.mark.parametrize("scan_mode", [0, 2, 3])
@pytest.mark.parametrize("residual", [False, True])
def test_workspaces_follow_the_calls(psb, mode, scan_mode, residual):
    """One session, calls that grow the buffers of one group at a time - queries, probes, results, candidate widths - and small ones between."""
    ix = synth.make_index(6000, 32, 1100, 8, seed=15, residual=residual)   # enough lists for the tensor-core coarse filter
    q = synth.make_queries(ix, 2500, seed=16)
    search = oracle.ivfrespq_search if residual else oracle.ivfpq_search
    with psb.Session(ix, n_rerank=60, exact_mode=mode, scan_mode=scan_mode, residual=residual, max_batch=2500) as s:
        for n, nprobe, k in ((1, 2, 5), (300, 2, 5), (7, 16, 5), (300, 2, 50), (2500, 2, 5), (2500, 16, 50), (3, 16, 50), (1200, 24, 55), (1, 1, 1)):
            got = s.search(q[:n], nprobe, k)
            lo = max(0, n - 40)
            want = search(ix, q[lo:n], nprobe, k, 60)
            assert np.array_equal(got["indices"][lo:], want["indices"]) and np.array_equal(got["distances"][lo:], want["distances"]), (n, nprobe, k)


def test_pool_goes_back_with_the_last_session(psb):
    """Training keeps its work memory in the library's pool; the last session of the device to end gives it back."""
    import torch
    ix = synth.make_index(2000, 32, 16, 8, seed=5)
    rows = torch.randn(600_000, 128, device="cuda")
    cen = rows[:1024].clone()
    assign = torch.empty(600_000, dtype=torch.int32, device="cuda")
    with psb.Session(ix, n_rerank=40, max_batch=64) as first:
        first.search(ix["vectors"][:1], 4, 10)
        second = psb.Session(ix, n_rerank=40, max_batch=64)
        psb.kmeans_train(rows, 600_000, 128, cen, 1024, 2, assign)
        torch.cuda.synchronize()
        kept = torch.cuda.mem_get_info()[0]
        second.close()
        assert abs(torch.cuda.mem_get_info()[0] - kept) < 32e6    # another session is there: the pool stays
    assert torch.cuda.mem_get_info()[0] - kept > 100e6             # 154 MB of operands alone
    psb.kmeans_train(rows, 600_000, 128, cen, 1024, 1, assign)     # and is taken anew
    torch.cuda.synchronize()
