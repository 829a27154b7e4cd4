"""The ADC scan's row form behind the stage calls: what a caller's batch and tables mean is what they mean to the other forms."""
import numpy as np
import pytest

import oracle
import synth

pytestmark = pytest.mark.gpu


def dev(a):
    import torch
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def outputs(nq, width):
    import torch
    return (torch.full((nq, width), -9, dtype=torch.int32, device="cuda"), torch.zeros((nq, width), device="cuda"),
            torch.zeros((nq,), dtype=torch.int32, device="cuda"))


@pytest.mark.parametrize("M,dim", [(48, 96), (20, 100)])   # with and without a tensor-core form
@pytest.mark.parametrize("residual", [False, True])
def test_empty_batch(psb, M, dim, residual):
    ix = synth.make_index(3000, dim, 8, M, seed=M, residual=residual)
    q = synth.make_queries(ix, 4, seed=1)
    probes, _ = oracle.coarse(q, ix["centroids"], 3)
    rows, dist, cnt = outputs(4, 20)
    with psb.Session(ix, residual=residual) as s:
        lut = dev(np.zeros((4 * 3 if residual else 4, M * 256), np.float32))
        s.stage_scan_queries(dev(q), lut, 0, dev(probes.astype(np.int32)), 3, 20, rows, dist, cnt)
        with pytest.raises(psb.PsbError):
            s.stage_scan_queries(dev(q), lut, -1, dev(probes.astype(np.int32)), 3, 20, rows, dist, cnt)
        s.sync()
    assert (rows.cpu().numpy() == -9).all()
