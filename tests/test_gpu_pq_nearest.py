"""Nearest codewords (psb_pq_encode) against the CPU checker: sub-vector lengths with one to four K steps of the filter, rows and
sub-quantisers that do not fill their tiles, fewer than 256 codewords, and ties, which the lowest code wins."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dim,M,K", [(1, 8, 4, 256), (255, 96, 48, 256), (513, 32, 8, 33), (300, 100, 20, 256), (1000, 96, 24, 255),
                                       (513, 30, 10, 64), (400, 128, 16, 256), (260, 100, 10, 256), (260, 96, 8, 100),
                                       (300, 64, 4, 256), (300, 66, 11, 40), (40000, 64, 16, 256)])
def test_encode_matches_checker(n, dim, M, K):
    import torch
    from paraselect_b200 import api
    rng = np.random.default_rng(n + dim + M)
    x = rng.standard_normal((n, dim)).astype(np.float32)
    cb = rng.standard_normal((M, K, dim // M)).astype(np.float32)
    cb[:, K // 2:] = cb[:, : K - K // 2]            # every codeword twice: exact ties
    x[: n // 3] = np.round(x[: n // 3] * 2) / 2     # a grid: ties between different codewords
    cb[0] = np.round(cb[0] * 2) / 2
    if n > 3:
        x[n // 2, 0], x[n // 2 + 1, 1] = np.nan, np.inf
    codes = torch.full((n, M), 99, dtype=torch.uint8, device="cuda")
    api.pq_encode(torch.from_numpy(x).cuda(), n, dim, torch.from_numpy(cb).cuda(), M, K, codes)
    torch.cuda.synchronize()
    assert np.array_equal(codes.cpu().numpy(), oracle.pq_encode(x, cb))
