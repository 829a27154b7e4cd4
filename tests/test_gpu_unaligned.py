"""Callers' device arrays that start at any float: queries and tables one element past an aligned address, in every form of the scan."""
import numpy as np
import pytest

import oracle
import synth

pytestmark = pytest.mark.gpu


def shifted(a):
    """The array on the device, one element past a 16-byte boundary."""
    import torch
    t = torch.from_numpy(np.ascontiguousarray(a))
    buf = torch.empty(t.numel() + 8, dtype=t.dtype, device="cuda")
    out = buf[1:1 + t.numel()].view(t.shape)
    out.copy_(t)
    assert out.data_ptr() % 16 == out.element_size()
    return out


@pytest.mark.parametrize("residual", [False, True])
@pytest.mark.parametrize("scan_mode", [0, 1, 2, 3])
@pytest.mark.parametrize("M,dim", [(48, 96), (8, 32), (16, 128)])
def test_scan_stage(psb, M, dim, scan_mode, residual):
    import torch
    nq, nprobe, width = 70, 4, 50
    ix = synth.make_index(9000, dim, 12, M, seed=M + 2, residual=residual)
    q = synth.make_queries(ix, nq, seed=2)
    probes, _ = oracle.coarse(q, ix["centroids"], nprobe)
    if residual:
        orow, odist, ocnt, _ = oracle.pq_scan_residual(q, probes, ix["centroids"], ix["offsets"], ix["codes"], ix["codebook"], width)
    else:
        orow, odist, ocnt, _ = oracle.pq_scan(q, probes, ix["offsets"], ix["codes"], ix["codebook"], width)
    dq, dp = shifted(q), shifted(probes.astype(np.int32))
    rows = shifted(np.zeros((nq, width), np.int32)); dist = shifted(np.zeros((nq, width), np.float32)); cnt = shifted(np.zeros(nq, np.int32))
    with psb.Session(ix, residual=residual, scan_mode=scan_mode) as s:
        lut = shifted(np.zeros((nq * (nprobe if residual else 1), M * 256), np.float32))
        (s.stage_build_lut_residual(dq, nq, dp, nprobe, lut) if residual else s.stage_build_lut(dq, nq, lut))
        s.stage_scan_queries(dq, lut, nq, dp, nprobe, width, rows, dist, cnt)
        s.sync()
        assert np.array_equal(rows.cpu().numpy(), orow) and np.array_equal(dist.cpu().numpy(), odist) and np.array_equal(cnt.cpu().numpy(), ocnt)
    with psb.Session(ix, n_rerank=40, residual=residual, scan_mode=scan_mode, max_batch=nq) as s:
        ids, d = torch.empty(nq, 10, dtype=torch.int64, device="cuda"), shifted(np.zeros((nq, 10), np.float32))
        s.search_device(dq, nq, nprobe, 10, ids, d)
        s.sync()
    want = (oracle.ivfrespq_search if residual else oracle.ivfpq_search)(ix, q, nprobe, 10, 40)
    assert np.array_equal(ids.cpu().numpy(), want["indices"]) and np.array_equal(d.cpu().numpy(), want["distances"])
