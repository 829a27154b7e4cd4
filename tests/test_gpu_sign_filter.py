"""Candidate search with float states where its tensor-core filter can go wrong: every word count, list lengths around the tiles (16,
64, 1,024 rows), states with one dominant, tiny or zero dimensions.  Rows and score bits equal the CPU checker's."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def dev(a):
    import torch
    a = np.ascontiguousarray(a)
    return torch.from_numpy(a.view(np.int32) if a.dtype == np.uint32 else a).cuda()


@pytest.mark.parametrize("padded", [32, 64, 128, 256])
@pytest.mark.parametrize("shape", ["normal", "dominant", "tiny", "zero"])
@pytest.mark.parametrize("nq,k", [(3, 1), (300, 40)])
def test_filter_keeps_every_candidate(psb, padded, shape, nq, k):
    import torch
    rng = np.random.default_rng(padded + nq)
    lengths = [1, 15, 16, 17, 63, 64, 65, 127, 129, 1023, 1024, 1025, 3000, 0, 2049]
    off = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int64)
    n, nlist, nprobe = int(off[-1]), len(lengths), 6
    codes = rng.integers(0, 2 ** 32, (n, padded // 32), dtype=np.uint64).astype(np.uint32)
    scales = (rng.random(n) + 0.25).astype(np.float32)
    probes = np.stack([np.r_[12, 14, rng.permutation(12)[:nprobe - 2]] for _ in range(nq)]).astype(np.int32)
    states = rng.standard_normal((nq * nprobe, padded)).astype(np.float32)
    if shape == "dominant":
        states[:, padded - 1] *= 1e4
    if shape == "tiny":
        states *= np.float32(1e-36)
    if shape == "zero":
        states[::2] = 0
    nsq = (states.astype(np.float64) ** 2).sum(1).astype(np.float32)
    rows = torch.empty((nq, k), dtype=torch.int32, device="cuda")
    dist = torch.empty((nq, k), dtype=torch.float32, device="cuda")
    psb.sign_search_candidates(0, dev(codes), dev(scales), dev(off), nlist, dev(probes), nq, nprobe, padded, k, rows, dist,
                               d_states=dev(states), d_norm_sq=dev(nsq))
    torch.cuda.synchronize()
    w_rows, w_dist = oracle.sign_candidates(0, codes, scales, off, probes, k, states=states, norm_sq=nsq)
    assert np.array_equal(rows.cpu().numpy(), w_rows)
    assert np.array_equal(dist.cpu().numpy().view(np.uint32), w_dist.view(np.uint32))
