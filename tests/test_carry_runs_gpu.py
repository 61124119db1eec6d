"""Rows that span many workers, bit for bit on integer-valued data: their carry records form runs
that end inside the 32 records of one warp, at its edge, one behind it and many warps on, and that
start at every place of a warp."""
import numpy as np
import pytest

import benchmark_spmv_using_csr_gb300 as sp
from benchmark_spmv_using_csr_gb300 import batch, gen

pytestmark = pytest.mark.gpu

PER_WORKER = 256  # 8 non-zeros per lane, one tile per worker


def matrix(workers, lead, n=3001):
    """`lead` workers of single-record rows, then one row per entry of `workers`, short rows
    between them."""
    lens = [PER_WORKER + 1] * lead
    for w in workers:
        lens += [PER_WORKER * w, 3, 0, 40]
    rp = np.zeros(len(lens) + 1, np.int64)
    rp[1:] = np.cumsum(lens)
    rng = np.random.default_rng(lead)
    col = rng.integers(0, n, rp[-1]).astype(np.int32)
    val = rng.integers(-3, 4, rp[-1]).astype(np.float64)
    return rp.astype(np.int32), col, val, n


@pytest.mark.parametrize("lead", [0, 1, 29, 31])
@pytest.mark.parametrize("workers", [(1, 2, 3, 2, 5), (30, 31, 32, 33), (64, 65, 96),
                                     (287, 288, 289, 320, 2)])
def test_runs_of_carry_records(cuda_ok, workers, lead):
    import torch
    rp, col, val, n = matrix(workers, lead)
    m = rp.size - 1
    x = np.random.default_rng(3).integers(-3, 4, (n, 8)).astype(np.float64)
    y = np.zeros((m, 8))
    np.add.at(y, np.repeat(np.arange(m), np.diff(rp)), val[:, None] * x[col])
    rpd, cid = torch.from_numpy(rp).cuda(), torch.from_numpy(col).cuda()
    for vt in (sp.VALUE_F64, sp.VALUE_F32, sp.VALUE_MIXED_F32):
        t = torch.float64 if vt == sp.VALUE_F64 else torch.float32
        p = sp.Plan(vt, m, n, rpd, cid, seg=8, tiles_per_worker=1, warps_per_cta=8, stages=0)
        p.set_grid(True)  # the tile kernel
        yd = torch.full((m,), float("nan"), dtype=t, device="cuda")
        p.execute(torch.from_numpy(val).cuda().to(t),
                  torch.from_numpy(np.ascontiguousarray(x[:, 0])).cuda().to(t), yd)
        p.check()
        np.testing.assert_array_equal(yd.cpu().double().numpy(), y[:, 0], err_msg=str(vt))
        p.close()
    for k in (1, 2, 8):
        b = batch.Batch([gen.CSR(m, n, rp, col, val)], k=k, seg=8, tiles_per_worker=1,
                        warps_per_cta=8)
        yd = torch.full((m, k), float("nan"), dtype=torch.float32, device="cuda")
        b.execute(torch.from_numpy(np.ascontiguousarray(x[:, :k])).cuda().float(), yd)
        b.check()
        np.testing.assert_array_equal(yd.cpu().double().numpy(), y[:, :k], err_msg=str(k))
        b.close()
