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


@pytest.mark.parametrize("n,dim,k", [(300, 64, 1024), (1000, 100, 1500), (64, 37, 2048), (65, 37, 128), (5000, 100, 131), (4097, 128, 255), (3000, 5, 256),
                                     (2500, 37, 257), (6000, 128, 511), (6000, 64, 512), (1025, 100, 513), (9000, 96, 700), (3333, 126, 1023)])
@pytest.mark.parametrize("prev", [None, "zeros", "far", "outside", "same"])
@pytest.mark.parametrize("form", [1, 2])
def test_either_form(psb, n, dim, k, prev, form):
    """The same through the form that is asked for, wherever the line between them lies: loose bounds, rows near nothing, ties, rows that are not
    numbers, centroids that fill a part of a block or a little of a second."""
    import torch
    g = torch.Generator(device="cuda"); g.manual_seed(n + dim + k)
    c = torch.randn(k, dim, device="cuda", generator=g)
    x = c[torch.randint(k, (n,), device="cuda", generator=g)] + 0.2 * torch.randn(n, dim, device="cuda", generator=g)
    x[1:20] = c[5] * 0.0
    x[20:30] = 40 * x[20:30]
    c[7] = c[6]
    c[k - 1] = c[3]
    x[30:40] = c[6]
    want_d, want = nearest(x, c)
    x[50, dim - 1], x[51, 0] = float("nan"), float("inf")
    fine = torch.ones(n, dtype=torch.bool, device="cuda"); fine[50:52] = False
    assign = {None: torch.full((n,), 77, dtype=torch.int32, device="cuda"), "zeros": torch.zeros(n, dtype=torch.int32, device="cuda"),
              "far": ((want + k // 2) % k).to(torch.int32), "outside": torch.full((n,), -1, dtype=torch.int32, device="cuda"),
              "same": want.to(torch.int32)}[prev].contiguous()
    best = torch.empty(n, device="cuda")
    psb.kmeans_assign(x, n, dim, c, k, assign, best, have_previous=prev is not None, form=form)
    assert torch.equal(best[fine], want_d[fine]) and torch.equal(assign.long()[fine], want[fine])
    assert bool(((assign >= 0) & (assign < k))[50:52].all())


def test_form_that_does_not_take_the_shape(psb):
    import torch
    x, c = torch.randn(100, 130, device="cuda"), torch.randn(200, 130, device="cuda")
    assign, best = torch.empty(100, dtype=torch.int32, device="cuda"), torch.empty(100, device="cuda")
    for n, dim, k in ((100, 130, 200), (63, 64, 200), (100, 64, 127)):
        with pytest.raises(psb.PsbError):
            psb.kmeans_assign(x, n, dim, c, k, assign, best, form=2)


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
