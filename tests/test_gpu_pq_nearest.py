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


@pytest.mark.parametrize("dim,M", [(8, 4), (16, 4), (32, 4), (20, 4), (64, 4)])   # two to sixteen dimensions a sub-vector
@pytest.mark.parametrize("scale", [3e18, 1e19, 1.8e19, 1e20])
def test_encode_where_products_overflow(dim, M, scale):
    """Magnitudes whose products pass the range of fp32 although distances to near codewords do not: rows are codewords or lie beside them."""
    import torch
    from paraselect_b200 import api
    rng = np.random.default_rng(dim)
    n, K = 700, 256
    cb = (rng.standard_normal((M, K, dim // M)) * scale).astype(np.float32)
    pick = rng.integers(0, K, (n, M))
    x = (cb[np.arange(M)[None, :], pick] * (1 + 1e-3 * rng.standard_normal((n, M, 1)))).astype(np.float32).reshape(n, dim)
    x[: n // 2] = cb[np.arange(M)[None, :], pick[: n // 2]].reshape(-1, dim)
    x[-20:] = 0.0
    codes = torch.full((n, M), 99, dtype=torch.uint8, device="cuda")
    api.pq_encode(torch.from_numpy(x).cuda(), n, dim, torch.from_numpy(cb).cuda(), M, K, codes)
    torch.cuda.synchronize()
    want = oracle.pq_encode(x, cb)
    assert np.array_equal(codes.cpu().numpy(), want)
    assert np.array_equal(want[: n // 2], pick[: n // 2])


@pytest.mark.parametrize("dim,M,K", [(8, 4, 100), (16, 4, 33), (32, 4, 255), (20, 4, 64), (64, 4, 40)])
@pytest.mark.parametrize("scale", [1e14, 1e16, 1e18, 1e19])
def test_encode_fewer_codewords_far_away(dim, M, K, scale):
    """Rows near the origin, fewer than 256 codewords all far from it: every score is a large negative number."""
    import torch
    from paraselect_b200 import api
    rng = np.random.default_rng(dim + K)
    n = 300
    cb = (np.sign(rng.standard_normal((M, K, dim // M))) * scale * (1 + 0.1 * rng.random((M, K, dim // M)))).astype(np.float32)
    x = (rng.standard_normal((n, dim)) * scale * 1e-3).astype(np.float32)
    x[: n // 3] = 0.0
    codes = torch.full((n, M), 99, dtype=torch.uint8, device="cuda")
    api.pq_encode(torch.from_numpy(x).cuda(), n, dim, torch.from_numpy(cb).cuda(), M, K, codes)
    torch.cuda.synchronize()
    assert np.array_equal(codes.cpu().numpy(), oracle.pq_encode(x, cb))


@pytest.mark.parametrize("dim,M", [(8, 4), (16, 4), (32, 4), (20, 4), (64, 4)])
@pytest.mark.parametrize("scale", [1e-16, 1e-18, 1e-19, 1e-20, 1e-22])
def test_encode_where_products_underflow(dim, M, scale):
    """Magnitudes whose products are subnormal or vanish: the filter's rounding is absolute there, not relative."""
    import torch
    from paraselect_b200 import api
    rng = np.random.default_rng(dim)
    n, K = 700, 256
    cb = (rng.standard_normal((M, K, dim // M)) * scale).astype(np.float32)
    x = (rng.standard_normal((n, dim)) * scale).astype(np.float32)
    codes = torch.full((n, M), 99, dtype=torch.uint8, device="cuda")
    api.pq_encode(torch.from_numpy(x).cuda(), n, dim, torch.from_numpy(cb).cuda(), M, K, codes)
    torch.cuda.synchronize()
    assert np.array_equal(codes.cpu().numpy(), oracle.pq_encode(x, cb))


@pytest.mark.parametrize("n,dim,M,K", [(127, 16, 4, 256), (128, 16, 5, 256), (129, 20, 5, 255), (1921, 24, 6, 256), (5000, 64, 16, 256), (70000, 8, 2, 256),
                                       (150, 400, 200, 40), (3000, 48, 4, 256), (2500, 33, 11, 33),
                                       (57600, 20, 5, 256), (113700, 20, 5, 256), (38000, 32, 16, 40)])   # items of nine and of fifteen tiles
@pytest.mark.parametrize("at", [0, 1, 2])
def test_encode_tiles_and_items(n, dim, M, K, at):
    """Rows at the ends of a tile and of an item's tiles, sub-quantisers that do not fill an operand row, rows that start at any float."""
    import torch
    from paraselect_b200 import api
    if dim % M:
        dim = dim // M * M
    rng = np.random.default_rng(n + dim + at)
    x = rng.standard_normal((n, dim)).astype(np.float32)
    cb = rng.standard_normal((M, K, dim // M)).astype(np.float32)
    flat = torch.empty(n * dim + 4, device="cuda")
    flat[at:at + n * dim] = torch.from_numpy(x).cuda().flatten()
    codes = torch.full((n * M + 4,), 99, dtype=torch.uint8, device="cuda")
    api.pq_encode(flat[at:at + n * dim], n, dim, torch.from_numpy(cb).cuda(), M, K, codes[at:at + n * M])
    torch.cuda.synchronize()
    got = codes.cpu().numpy()
    assert np.array_equal(got[at:at + n * M].reshape(n, M), oracle.pq_encode(x, cb))
    assert (got[:at] == 99).all() and (got[at + n * M:] == 99).all()


@pytest.mark.parametrize("n,dim,M,K,items", [
    (20000, 64, 16, 256, 0), (20000, 64, 16, 256, 50),      # 108 items, a block each: two turns of three tiles
    (200000, 64, 16, 256, 0), (200000, 64, 16, 256, 149), (200000, 64, 16, 256, 419),   # 420 items: no product, some or nearly all before the wait
    (300, 64, 4, 40, 0), (5000, 96, 24, 255, 1), (700, 32, 4, 256, 1)])
def test_encode_when_a_wait_gives_up(n, dim, M, K, items):
    """The time-out path: blocks whose items get no products wait for them until the limit; they then wait for the products they have issued,
    free their tensor memory and evaluate their rows without the filter.  The codes are the same, the device stays usable."""
    import torch
    from paraselect_b200 import api
    rng = np.random.default_rng(n + items)
    x = rng.standard_normal((n, dim)).astype(np.float32)
    cb = rng.standard_normal((M, K, dim // M)).astype(np.float32)
    want = oracle.pq_encode(x, cb)
    dx, dcb, gave_up = torch.from_numpy(x).cuda(), torch.from_numpy(cb).cuda(), torch.zeros(1, dtype=torch.int32, device="cuda")
    for few in (items, -1):
        codes = torch.full((n, M), 99, dtype=torch.uint8, device="cuda")
        gave_up.zero_()
        torch.cuda.synchronize()
        api.pq_encode_limited(dx, n, dim, dcb, M, K, codes, items=few, d_gave_up=gave_up)
        torch.cuda.synchronize()
        assert np.array_equal(codes.cpu().numpy(), want)
        assert (int(gave_up) > 0) == (few >= 0)
