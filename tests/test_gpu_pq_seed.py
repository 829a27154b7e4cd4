"""Seeding of the PQ trainer on the device against the host's k-means++ (psb_kmeans_init, itself pinned to the reference's draws): the
same rows, with fewer rows than codewords, rows that repeat (the distances run out and the host takes over), sub-vectors that fit the
kernel's shared memory and ones that do not, values that are not numbers, and the random-rows policy of large sets."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,dim,M,K,kind", [(3000, 16, 4, 256, "normal"), (70001, 16, 2, 256, "normal"), (5000, 10, 2, 256, "normal"),
                                            (4097, 12, 6, 255, "normal"), (100, 8, 2, 256, "normal"), (7, 8, 2, 4, "normal"),
                                            (2000, 16, 4, 256, "repeats"), (2000, 16, 4, 64, "grid"), (500, 8, 2, 16, "nan"),
                                            (60000, 48, 2, 128, "normal"), (90000, 8, 2, 256, "normal"), (1, 4, 1, 256, "normal")])
def test_first_codewords_are_the_hosts(psb, n, dim, M, K, kind):
    import torch
    rng = np.random.default_rng(n + dim)
    x = rng.standard_normal((n, dim)).astype(np.float32)
    if kind == "repeats":
        x = x[rng.integers(0, 50, n)]
    if kind == "grid":
        x = rng.integers(0, 4, (n, dim)).astype(np.float32)
    if kind == "nan":
        x[n // 2, 1] = np.nan
    cb = torch.empty((M, K, dim // M), dtype=torch.float32, device="cuda")
    psb.pq_train(torch.from_numpy(x).cuda(), n, dim, M, K, 0, 1234, cb)
    got = cb.cpu().numpy()
    d = dim // M
    for s in range(M):
        want, _ = psb.kmeans_init(np.ascontiguousarray(x[:, s * d:(s + 1) * d]), K, 1234 + s * 104729)
        assert np.array_equal(got[s].view(np.uint32), want.view(np.uint32)), "subspace %d" % s
