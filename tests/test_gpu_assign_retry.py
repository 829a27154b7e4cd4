"""Nearest-centroid assignment where the bound a row brings along is no help: the rows that fail are gathered and searched again with
two passes; rows that fail there too (a value that is not a number) get the exact kernel.  And codeword groups above 1,024 rows in the
accumulation.  Against plain fp32 arithmetic in the same order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def nearest(x, c):
    import torch
    d = torch.zeros(x.shape[0], c.shape[0], device="cuda")
    for j in range(x.shape[1]):   # sequential, non-fused
        t = x[:, j:j + 1] - c[:, j][None, :]
        d = d + t * t
    return d.min(1).values, d.argmin(1)


@pytest.mark.parametrize("n,dim,k", [(300, 64, 1024), (1000, 100, 1500), (70001, 128, 1024), (64, 37, 2048)])
@pytest.mark.parametrize("prev", ["zeros", "far", "outside"])
def test_useless_bounds(psb, n, dim, k, prev):
    import torch
    g = torch.Generator(device="cuda"); g.manual_seed(n + dim)
    c = torch.randn(k, dim, device="cuda", generator=g)
    x = c[torch.randint(k, (n,), device="cuda", generator=g)] + 0.2 * torch.randn(n, dim, device="cuda", generator=g)
    x[1:20] = c[5] * 0.0                                        # rows near nothing: long candidate lists
    c[7] = c[6]                                                 # a tie: the lower id wins
    want_d, want = nearest(x, c)
    assign = {"zeros": torch.zeros(n, dtype=torch.int32, device="cuda"), "far": ((want + k // 2) % k).to(torch.int32),
              "outside": torch.full((n,), -1, dtype=torch.int32, device="cuda")}[prev].contiguous()
    best = torch.empty(n, device="cuda")
    psb.kmeans_assign(x, n, dim, c, k, assign, best, have_previous=True)
    assert torch.equal(best, want_d) and torch.equal(assign.long(), want)
    psb.kmeans_assign(x, n, dim, c, k, assign, best)            # the two passes without a bound
    assert torch.equal(best, want_d) and torch.equal(assign.long(), want)


@pytest.mark.parametrize("n,dim,k,big", [(5000, 128, 40, 3000), (9000, 100, 7, 1025), (1024, 33, 1, 1024), (2000, 300, 5, 1500)])
def test_sums_of_large_groups(psb, n, dim, k, big):
    import torch
    g = torch.Generator(device="cuda"); g.manual_seed(n)
    x = torch.randn(n, dim, device="cuda", generator=g)
    a = torch.randint(k, (n,), device="cuda", generator=g, dtype=torch.int32)
    a[:big] = 0
    best = torch.rand(n, device="cuda", generator=g)
    sums = torch.empty(k, dim, dtype=torch.float64, device="cuda")
    counts = torch.empty(k, dtype=torch.int32, device="cuda")
    obj = torch.empty(1, dtype=torch.float64, device="cuda")
    psb.kmeans_accumulate(x, n, dim, a, best, k, sums, counts, obj)
    one = torch.zeros(k, n, dtype=torch.float64, device="cuda")
    one[a.long(), torch.arange(n, device="cuda")] = 1.0
    assert torch.equal(counts.long(), one.sum(1).long())
    assert np.allclose(sums.cpu().numpy(), (one @ x.double()).cpu().numpy(), rtol=1e-12, atol=1e-9)
    assert abs(float(obj) - float(best.double().sum())) < 1e-6
