"""k-means on few centroids: the nearest of them by rows and, above the line of work, by the filter; counts and places by blocks of rows."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def distances(x, c):
    d = np.zeros((len(x), len(c)), np.float32)
    for j in range(x.shape[1]):   # in the order of the dimensions, nothing fused
        t = x[:, None, j] - c[None, :, j]
        d += t * t
    return d


@pytest.mark.parametrize("n,dim,k", [(1, 8, 1), (63, 8, 1), (64, 5, 64), (65, 33, 65), (4096, 20, 63), (4097, 12, 129), (300, 200, 70), (8193, 3, 7),
                                     (5000, 48, 700), (3000, 130, 300), (20000, 16, 2049), (12289, 8, 2048),
                                     # few rows: centroids in ranges, or a thread for each pair; long rows and many centroids
                                     (1, 100, 3000), (40, 16, 900), (51, 128, 1000), (701, 64, 1500), (9001, 20, 321), (2047, 200, 513), (2049, 200, 513),
                                     # both sides of the line to counts by blocks of rows
                                     (16383, 8, 512), (16384, 8, 512), (16385, 8, 513), (20481, 5, 1), (33000, 6, 1031),
                                     # above the line to the filter, whose blocks are of 512 centroids
                                     (20000, 128, 200), (30000, 100, 300), (24001, 128, 511)])
@pytest.mark.parametrize("odd", [False, True])
def test_assignment_and_means(psb, n, dim, k, odd):
    import torch
    rng = np.random.default_rng(n + k)
    x = rng.integers(-3, 4, (n, dim)).astype(np.float32) if n % 2 else rng.standard_normal((n, dim)).astype(np.float32)   # a grid: ties
    c = x[rng.integers(0, n, k)] + (0 if n % 2 else 0.1 * rng.standard_normal((k, dim)).astype(np.float32))
    if odd and n > 64:
        x[n // 2, 0], x[n // 3, dim - 1] = np.inf, np.nan
    c = c.astype(np.float32)
    d = distances(x, c)
    want = np.where(np.isnan(d), np.float32(np.inf), d).argmin(1)
    dx, cen, assign = torch.from_numpy(x).cuda(), torch.from_numpy(c).cuda(), torch.empty(n, dtype=torch.int32, device="cuda")
    psb.kmeans_train(dx, n, dim, cen, k, 0, assign)
    torch.cuda.synchronize()
    got = assign.cpu().numpy()
    fine = np.isfinite(d).any(1)
    assert np.array_equal(got[fine], want[fine]) and (got >= 0).all() and (got < k).all()
    if odd:
        return
    psb.kmeans_train(dx, n, dim, cen, k, 1, assign)
    torch.cuda.synchronize()
    new = cen.cpu().numpy()
    for i in np.unique(rng.integers(0, k, 40)):
        mean = x[want == i].astype(np.float64).mean(0) if (want == i).any() else c[i]
        assert np.allclose(new[i], mean, rtol=1e-6, atol=1e-6)      # fp64 sums, rounded once
