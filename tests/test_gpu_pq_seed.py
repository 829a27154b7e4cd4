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


@pytest.mark.parametrize("n,dim,M,K", [(2049, 15, 5, 256), (8193, 30, 6, 200), (600, 18, 3, 256), (32769, 20, 4, 256), (4095, 8, 4, 256), (8192, 16, 4, 256), (600, 8, 2, 256),
                                       (68256, 10, 2, 256), (45504, 16, 2, 256)])   # the most rows that shared memory holds
def test_stretches_of_the_search(psb, n, dim, M, K):
    """Sub-vectors of two, three, five and six; stretches that end within a lane's eight rows; both searches at the line between them."""
    test_first_codewords_are_the_hosts(psb, n, dim, M, K, "normal")


@pytest.mark.parametrize("n,dim,M,K", [(4097, 15, 5, 256), (300, 20, 4, 100), (9000, 24, 2, 64), (5000, 80, 2, 40), (4096, 6, 3, 256), (700, 3, 3, 256)])
def test_codewords_are_the_means_of_their_rows(psb, n, dim, M, K):
    """One iteration from the first codewords: sub-vectors of one to forty dimensions, row ranges that do not fill a block."""
    import torch
    rng = np.random.default_rng(n + dim)
    x = rng.standard_normal((n, dim)).astype(np.float32)
    d, dx = dim // M, torch.from_numpy(x).cuda()
    first, then = (torch.empty((M, K, d), dtype=torch.float32, device="cuda") for _ in range(2))
    psb.pq_train(dx, n, dim, M, K, 0, 7, first)
    psb.pq_train(dx, n, dim, M, K, 1, 7, then)
    f, got = first.cpu().numpy().astype(np.float64), then.cpu().numpy()
    for s in range(M):
        xs = x[:, s * d:(s + 1) * d].astype(np.float64)
        near = ((xs[:, None, :] - f[s][None]) ** 2).sum(2).argmin(1)
        for c in range(K):
            want = xs[near == c].mean(0) if (near == c).any() else f[s][c]
            assert np.allclose(got[s][c], want, rtol=1e-6, atol=1e-6)      # fp64 sums, rounded once: 6e-8 of values up to 4
