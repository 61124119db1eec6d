"""The row kernel and the batch's work lists beyond exact integers on small cases: random shapes and
values, Inf and NaN, FP64 layouts, and non-zeros near 2^31."""
import ctypes

import numpy as np
import pytest

import oracle
from conftest import TOL_F32, TOL_F64, TOL_MIXED_NORMWISE

import benchmark_spmv_using_csr_gb300 as sp
from benchmark_spmv_using_csr_gb300 import batch
from benchmark_spmv_using_csr_gb300._lib import lib

pytestmark = pytest.mark.gpu

VTS = [sp.VALUE_F64, sp.VALUE_F32, sp.VALUE_MIXED_F32, sp.VALUE_MIXED_BF16]
MAX_NNZ = 2147479551  # BHSP_MAX_NNZ of include/spmv_gb300.h


def even_rows(rng, vt):
    """Rows whose lengths differ by little, so that they fill their lanes' slots: the row kernel."""
    m = int(np.exp(rng.uniform(0, np.log(60_000))))
    top = int(rng.integers(1, 33 if vt == sp.VALUE_F64 else 225))
    if top > 56:
        m = min(m, 8000)
    # the whole slots of the layout's groups of 4 that the longest row takes
    lanes = 1
    while top > 28 * lanes:
        lanes *= 2
    low = max(1, int(0.9 * -(-top // (4 * lanes)) * 4 * lanes))
    lens = rng.integers(min(low, top), top + 1, m)
    n = int(rng.integers(max(top, 1), 3 * m + top + 1))
    lens[rng.random(m) < rng.choice([0.0, 0.02])] = 0
    rp = np.zeros(m + 1, np.int32)
    rp[1:] = np.cumsum(lens)
    row = np.repeat(np.arange(m), lens)
    if rng.integers(0, 2):  # near columns
        col = (row + np.arange(row.size) - rp[row]) % n
    else:
        col = rng.integers(0, n, row.size)
    return rp, col.astype(np.int32), n


def run(torch, vt, rp, col, n, val, x):
    """(y as float64, whether the row kernel ran)"""
    store = {sp.VALUE_F64: torch.float64, sp.VALUE_MIXED_BF16: torch.bfloat16}.get(vt, torch.float32)
    vec = torch.float64 if vt == sp.VALUE_F64 else torch.float32
    m = rp.size - 1
    col = col if col.size else np.zeros(8, np.int32)
    vd = torch.from_numpy(val if val.size else np.zeros(8)).cuda().to(store)
    xd = torch.from_numpy(x).cuda().to(vec)
    y = torch.full((m,), float("nan"), dtype=vec, device="cuda")
    p = sp.Plan(vt, m, n, torch.from_numpy(rp).cuda(), torch.from_numpy(col).cuda(), nnz=int(rp[-1]))
    rows = p.kernel()[0] > 0
    for _ in range(2):
        p.execute(vd, xd, y)
    p.check()
    p.close()
    return y.cpu().double().numpy(), rows


@pytest.mark.parametrize("vt", VTS)
def test_random_even_rows(cuda_ok, vt):
    """Real values against the compensated oracle, at the stated tolerances; most draws take the row
    kernel, in FP64 a third."""
    import torch
    rng = np.random.default_rng(50 + vt)
    took = 0
    for i in range(60):
        rp, col, n = even_rows(rng, vt)
        val, x = rng.uniform(-1, 1, col.size), rng.uniform(-1, 1, n)
        if vt != sp.VALUE_F64:
            val, x = val.astype(np.float32).astype(np.float64), x.astype(np.float32).astype(np.float64)
        if vt == sp.VALUE_MIXED_BF16:
            val = torch.from_numpy(val).to(torch.bfloat16).double().numpy()
        y, rows = run(torch, vt, rp, col, n, val, x)
        took += rows
        want = oracle.csr_dot2(rp, col, val, x)
        if vt in (sp.VALUE_F64, sp.VALUE_F32):
            scale = oracle.csr_absrow(rp, col, val, x)
            tol = TOL_F64 if vt == sp.VALUE_F64 else TOL_F32
            assert oracle.componentwise_error(y, want, scale) <= tol, (i, rp.size, n)
        elif np.linalg.norm(want) > 0:
            assert oracle.normwise_error(y, want) <= TOL_MIXED_NORMWISE, (i, rp.size, n)
    # (FP64 asks for 0.84 of the slots, which longest rows of 5, 9, 13, ... leave unfilled)
    assert took >= (20 if vt == sp.VALUE_F64 else 40), took


@pytest.mark.parametrize("vt", VTS)
def test_inf_and_nan_in_the_row_kernel(cuda_ok, vt):
    """Inf and NaN in x and in the values reach exactly the rows of the serial loop (the compensated
    forms turn an infinite row into NaN); every finite row is exact."""
    import torch
    rng = np.random.default_rng(9 + vt)
    took = 0
    for i in range(12):
        rp, col, n = even_rows(rng, vt)
        if col.size < 2000 or n < 100:
            continue
        val, x = rng.integers(-4, 5, col.size).astype(float), rng.integers(-4, 5, n).astype(float)
        x[rng.choice(n, 3, replace=False)] = [np.inf, -np.inf, np.nan]
        val[rng.choice(val.size, 3, replace=False)] = [np.inf, -np.inf, np.nan]
        want = oracle.csr_serial(rp, col, val, x)
        y, rows = run(torch, vt, rp, col, n, val, x)
        took += rows
        fin = np.isfinite(want)
        assert (y[fin] == want[fin]).all()
        if vt in (sp.VALUE_F64, sp.VALUE_F32):
            np.testing.assert_array_equal(y[~fin], want[~fin])
        else:
            assert not np.isfinite(y[~fin]).any()
    assert took >= 5


@pytest.mark.parametrize("m", [1, 33, 1001])
def test_fp64_layouts_take_the_row_kernel(cuda_ok, m):
    """FP64 rows of 29 to 32 non-zeros: two lanes to a row."""
    import torch
    for top in (29, 30, 31, 32):
        rp = np.arange(0, (m + 1) * top, top, dtype=np.int32)
        col = ((np.arange(m * top) // top + np.arange(m * top) % top) % m).astype(np.int32)
        p = sp.Plan(sp.VALUE_F64, m, m, torch.from_numpy(rp).cuda(), torch.from_numpy(col).cuda())
        # one lane's passes are whole at 32 rows, two lanes' at 16: a few rows alone fill too little
        assert p.kernel() == ((2, 16) if m * top >= 0.84 * 128 * -(-m // 16) * 4 else (0, 0)), top
        p.close()


def integer_batch(rng, k):
    from benchmark_spmv_using_csr_gb300 import gen
    lens = rng.integers(0, 40, 700)
    lens[[5, 300, 690]] = [2500, 225, 1111]
    mats = [gen.from_row_lengths(np.asarray(l), 3000, seed=int(rng.integers(1 << 30))) for l in (
        np.full(6001, 27), lens, np.full(1024, 5), rng.integers(240, 900, 300), np.full(6000, 32),
        rng.integers(100, 113, 256))]
    for a in mats:
        a.val = rng.integers(-4, 5, a.nnz).astype(np.float64)
    return batch.Batch(mats, k=k)


@pytest.mark.parametrize("k", [1, 2, 4, 8])
def test_inf_and_nan_in_work_lists(cuda_ok, k):
    """As in the row kernel, per right-hand side: an Inf or NaN in one leaves the others exact."""
    import torch
    rng = np.random.default_rng(31 + k)
    b = integer_batch(rng, k)
    assert b.info()["row_lists"] > 0 and b.info()["tile_workers"] > 0
    x = rng.integers(-4, 5, (b.n, k)).astype(np.float64)
    for j in range(k):
        x[rng.choice(b.n, 6, replace=False), j] = [np.inf, -np.inf, np.nan] * 2
    cat = b.cat
    want = np.stack([oracle.csr_serial(cat["row_ptr"], cat["col"], cat["val"], x[:, j].copy())
                     for j in range(k)], 1)
    assert not np.isfinite(want).all() and np.isfinite(want).any()
    y = torch.empty((b.m, k), dtype=torch.float32, device="cuda")
    xd = torch.from_numpy(x.astype(np.float32)).cuda()
    for _ in range(2):
        y.fill_(0.0)
        b.execute(xd, y)
        b.check()
        yh = y.cpu().double().numpy()
        fin = np.isfinite(want)
        assert (yh[fin] == want[fin]).all() and not np.isfinite(yh[~fin]).any()
    b.close()


N = 1_000_003


@pytest.fixture(scope="module")
def big(cuda_ok):
    """MAX_NNZ non-zeros: rows of 200 (the row kernel), then, for the batch, a last run of rows of
    1000 to 2200 whose windows lie at the end."""
    import torch
    dev = "cuda"
    j = torch.arange(MAX_NNZ, device=dev, dtype=torch.int64)
    col = ((j * 7919) % N).to(torch.int32)
    small = (j % 5).to(torch.uint8)
    del j
    x = (torch.arange(N, device=dev, dtype=torch.int64) % 3).to(torch.uint8)
    prod = small * x[col.long()]
    sums = torch.zeros(MAX_NNZ + 1, device=dev, dtype=torch.int64)
    torch.cumsum(prod, 0, dtype=torch.int64, out=sums[1:])
    del prod
    torch.cuda.empty_cache()
    yield col, small, x, sums
    del sums
    torch.cuda.empty_cache()


def big_rows(torch, lens):
    ends = torch.cumsum(lens, 0).clamp(max=MAX_NNZ)
    m = int(torch.searchsorted(ends, torch.tensor([MAX_NNZ], device="cuda")).item()) + 1
    rp = torch.zeros(m + 1, device="cuda", dtype=torch.int64)
    rp[1:] = ends[:m]
    assert int(rp[-1]) == MAX_NNZ
    return m, rp


@pytest.mark.parametrize("vt", [sp.VALUE_F32, sp.VALUE_MIXED_BF16])
def test_max_nnz_row_kernel(big, vt):
    import torch
    col, small, x, sums = big
    m, rp = big_rows(torch, torch.full((MAX_NNZ // 200 + 2,), 200, device="cuda", dtype=torch.int64))
    val = small.to(torch.bfloat16 if vt == sp.VALUE_MIXED_BF16 else torch.float32)
    y = torch.full((m,), -1.0, device="cuda")
    p = sp.Plan(vt, m, N, rp.to(torch.int32), col)
    assert p.kernel() == (8, 28)
    p.execute(val, x.float(), y)
    p.check()
    p.close()
    assert bool((y.double() == (sums[rp[1:]] - sums[rp[:-1]]).double()).all())


@pytest.mark.parametrize("k,rows", [(1, 100), (2, 200)])
def test_max_nnz_work_lists(big, k, rows):
    import torch
    col, small, x, sums = big
    even = torch.full((int(0.9 * MAX_NNZ) // rows,), rows, device="cuda", dtype=torch.int64)
    i = torch.arange(200_000, device="cuda", dtype=torch.int64)
    long_rows = torch.where(i % 7 == 3, torch.zeros_like(i), 1000 + (i % 5) * 300)
    m, rp = big_rows(torch, torch.cat([even, long_rows]))
    val = small.float()
    xs = torch.stack([x.float() * (j + 1) for j in range(k)], 1).contiguous()
    y = torch.full((m, k), -1.0, device="cuda")
    rp32, L, b = rp.to(torch.int32), lib(), ctypes.c_void_p()
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    assert L.bhsp_batch_create(ctypes.byref(b), 1, m, N, MAX_NNZ, rp32.data_ptr(), col.data_ptr(), k, 0,
                               0, 0, stream) == 0
    lists, workers = ctypes.c_int(), ctypes.c_int()
    L.bhsp_batch_lists(b, ctypes.byref(lists), ctypes.byref(workers), None, None)
    assert lists.value > 0 and workers.value > 0
    assert L.bhsp_batch_execute(b, val.data_ptr(), xs.data_ptr(), y.data_ptr(), 0, stream) == 0
    assert L.bhsp_batch_check(b, stream) == 0
    L.bhsp_batch_destroy(b)
    want = (sums[rp[1:]] - sums[rp[:-1]]).double()
    for j in range(k):
        assert bool((y[:, j].double() == want * (j + 1)).all()), j
