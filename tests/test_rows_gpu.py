"""The row kernel (lanes assigned to whole rows), which a plan takes for matrices whose rows are
short and fill their lanes' slots: bit for bit against an int64
sum on integer-valued data, at the edges of its lane layouts (1 to 8 lanes per row, 1 to 7 groups
of 4 slots each), of its passes of 32 lanes and of the bulk copies' groups of 8 non-zeros."""
import numpy as np
import pytest

import benchmark_spmv_using_csr_gb300 as sp

pytestmark = pytest.mark.gpu

VTS = [sp.VALUE_F64, sp.VALUE_F32, sp.VALUE_MIXED_F32, sp.VALUE_MIXED_BF16]
# longest row: 1 lane up to 28, 2 up to 56, 4 up to 112, 8 up to 224; FP64 up to 32
LENGTHS = [1, 4, 5, 8, 9, 12, 13, 16, 17, 20, 24, 25, 28, 29, 32, 33, 48, 56, 57, 64, 112, 113, 224]


def banded(torch, lens, seed):
    """Rows of the given lengths whose columns run on from the row's number (modulo m)."""
    m = lens.size
    rp = np.zeros(m + 1, np.int32)
    rp[1:] = np.cumsum(lens)
    row = np.repeat(np.arange(m), lens)
    col = ((row + np.arange(row.size) - rp[row]) % m).astype(np.int32)
    rng = np.random.default_rng(seed)
    val = rng.integers(-4, 5, row.size).astype(np.float64)
    x = rng.integers(-4, 5, m).astype(np.float64)
    y = np.zeros(m)
    np.add.at(y, row, val * x[col])
    return rp, col, val, x, y


def device(torch, vt, a):
    store = {sp.VALUE_F64: torch.float64, sp.VALUE_MIXED_BF16: torch.bfloat16}.get(vt, torch.float32)
    vec = torch.float64 if vt == sp.VALUE_F64 else torch.float32
    rp, col, val, x, _ = a
    return (torch.from_numpy(rp).cuda(), torch.from_numpy(col).cuda(),
            torch.from_numpy(val).cuda().to(store), torch.from_numpy(x).cuda().to(vec),
            torch.full((x.size,), float("nan"), dtype=vec, device="cuda"))


@pytest.mark.parametrize("vt", VTS)
@pytest.mark.parametrize("m", [1, 3, 31, 32, 33, 1001])
def test_lane_layouts_bit_exact(cuda_ok, vt, m):
    """Every layout, with all rows at the longest length and with some shorter and empty ones (at
    the start, the end and between), twice: y must not depend on what it held."""
    import torch
    for top in LENGTHS:
        whole = np.full(m, top)
        mixed = whole.copy()
        mixed[m // 2::7] -= min(2, top - 1)
        mixed[3::50] = 0
        if m > 1000:
            mixed[:2] = mixed[-40:] = 0
        for lens in (whole, mixed):
            a = banded(torch, lens, 10 * top + m)
            rp, col, val, x, y = device(torch, vt, a)
            p = sp.Plan(vt, m, m, rp, col)
            if vt != sp.VALUE_F64 and m > 1000 and top not in (1, 5, 9, 13):
                assert p.launches == 1, (top, "the row kernel")
            for _ in range(2):
                p.execute(val, x, y)
                p.check()
                bad = int((y.cpu().double().numpy() != a[4]).sum())
                assert bad == 0, (top, bad)
                y.fill_(float("nan"))
            p.close()


@pytest.mark.parametrize("vt", VTS)
def test_many_passes_per_warp_bit_exact(cuda_ok, vt):
    """More passes than warps: the strided workers, and for FP64 the ticket, whose last warp leaves
    it at zero for the next launch.  A forced variant or grid sends the same plan to the tile
    kernel, with the same y."""
    import torch
    m = 900_001
    lens = np.full(m, 27)
    lens[::160] = lens[159::160] = 18
    a = banded(torch, lens, 5)
    rp, col, val, x, y = device(torch, vt, a)
    p = sp.Plan(vt, m, m, rp, col)
    assert p.launches == 1
    want = torch.from_numpy(a[4]).cuda().to(y.dtype)
    for _ in range(3):
        y.fill_(float("nan"))
        p.execute(val, x, y)
        p.check()
        assert torch.equal(y, want)
    p.set_grid(False)
    assert p.launches == 2
    y.fill_(float("nan"))
    p.execute(val, x, y)
    p.check()
    assert torch.equal(y, want)
    p.set_grid(None)
    assert p.launches == 1
    p.set_variant(l2_only=False)
    assert p.launches == 2
    p.close()


def test_row_kernel_decision(cuda_ok):
    """Short rows that fill their slots take the row kernel: 0.6 of them with near columns, a third
    with random ones, 0.84 in FP64; one long row sends the matrix to the tile kernels."""
    import torch
    rng = np.random.default_rng(1)

    def launches(lens, vt=sp.VALUE_F32, spread=False):
        rp, col = banded(torch, lens, 2)[:2]
        if spread:
            col = rng.integers(0, lens.size, col.size).astype(np.int32)
        p = sp.Plan(vt, lens.size, lens.size, torch.from_numpy(rp).cuda(), torch.from_numpy(col).cuda())
        try:
            return p.launches
        finally:
            p.close()

    m = 20_000
    whole = np.full(m, 27)
    assert launches(whole) == 1 and launches(whole, sp.VALUE_F64) == 1
    assert launches(whole, spread=True) == 1 and launches(whole, sp.VALUE_F64, spread=True) == 1
    one_long = whole.copy()
    one_long[77] = 225
    assert launches(one_long) == 2
    assert launches(np.full(m, 33), sp.VALUE_F64) == 2 and launches(np.full(m, 33)) == 1
    uneven = rng.integers(0, 28, m)  # half of the 28 slots on average
    assert launches(uneven) == 2 and launches(uneven, spread=True) == 1
    assert launches(uneven, sp.VALUE_F64, spread=True) == 2
    three_quarters = rng.integers(20, 28, m)  # 24 of 28 slots on average
    assert launches(three_quarters) == 1


@pytest.mark.parametrize("k", [1, 2, 4, 8])
@pytest.mark.parametrize("seg", [8, 16, 32])
def test_batch_work_lists_bit_exact(cuda_ok, k, seg):
    """The batched form's row and tile workers in one batch: runs of long rows that begin and end
    inside a tile, between blocks of every row layout; empty rows at the start and end of a run
    and of the batch, an all-empty member, a last block of a few rows, non-zeros not a multiple of
    8; run twice, and against the one tile kernel (a forced variant)."""
    import torch
    from benchmark_spmv_using_csr_gb300 import batch, gen
    rng = np.random.default_rng(10 * k + seg)

    def rows(lens):
        a = gen.from_row_lengths(np.asarray(lens), 3000, seed=int(rng.integers(1 << 30)))
        a.val = rng.integers(-4, 5, a.nnz).astype(np.float64)
        return a

    long_rows = rng.integers(0, 40, 700)
    long_rows[[5, 300, 690]] = [2500, 225, 1111]
    long_rows[:4] = long_rows[-3:] = 0
    mats = [rows(np.zeros(300, int)), rows(np.full(6001, 27)), rows(long_rows),
            rows(np.full(260, 32)), rows(np.full(1024, 5)), rows(rng.integers(50, 57, 256)),
            rows(long_rows[::-1]), rows(rng.integers(100, 113, 256)),
            rows(rng.integers(200, 225, 256)), rows(np.full(3, 7))]
    b = batch.Batch(mats, k=k, seg=seg)
    info = b.info()
    # tile workers, one lane layout for all row blocks (there are few), the carry records (at k = 1 a
    # kernel of their own)
    assert info["launches"] in ((3, 4) if k == 1 else (2, 3))
    x_np = rng.integers(-4, 5, (b.n, k)).astype(np.float64)
    cat = b.cat
    row = np.repeat(np.arange(b.m), np.diff(cat["row_ptr"]))
    want = np.zeros((b.m, k))
    np.add.at(want, row, cat["val"][:, None] * x_np[cat["col"]])
    x = torch.from_numpy(x_np.astype(np.float32)).cuda()
    y = torch.empty((b.m, k), dtype=torch.float32, device="cuda")
    grids = set()
    for l2 in (None, None, True):
        b.set_variant(l2_only=l2)
        grids.add(b.info()["grid"])
        for use_graph in (True, False):
            y.fill_(float("nan"))
            b.execute(x, y, use_graph=use_graph)
            b.check()
            assert (y.cpu().numpy() == want).all(), (l2, use_graph)
    b.close()


@pytest.mark.parametrize("k", [1, 2, 4, 8])
def test_batch_row_lists_bit_exact(cuda_ok, k):
    """Every list of row blocks: members large enough for a kernel per lane
    layout, a ragged last block, with and without runs of long rows between them."""
    import torch
    from benchmark_spmv_using_csr_gb300 import batch, gen
    rng = np.random.default_rng(77)
    regular = [np.full(160_000, 5), rng.integers(11, 17, 160_000), np.full(80_005, 27),
               np.full(80_000, 32), rng.integers(50, 57, 40_100), np.full(40_001, 112)]
    if k == 1:  # 2 layouts of 2 lanes (1 to 8 and 9 to 28 slots would be one elsewhere), none of 8
        lists = 6
    else:
        regular.append(rng.integers(220, 225, 20_001))
        lists = 5
    long_rows = np.full(600, 300)
    for parts, launches in ((regular, lists),
                            (regular[:3] + [long_rows] + regular[3:], lists + (2 if k == 1 else 1))):
        mats = []
        for lens in parts:
            a = gen.from_row_lengths(lens, 5000, seed=int(rng.integers(1 << 30)))
            a.val = rng.integers(-4, 5, a.nnz).astype(np.float64)
            mats.append(a)
        b = batch.Batch(mats, k=k)
        assert b.info()["launches"] == launches
        x_np = rng.integers(-4, 5, (b.n, k)).astype(np.float64)
        row = np.repeat(np.arange(b.m), np.diff(b.cat["row_ptr"]))
        want = np.stack([np.bincount(row, b.cat["val"] * x_np[b.cat["col"], i], b.m)
                         for i in range(k)], 1)
        x = torch.from_numpy(x_np.astype(np.float32)).cuda()
        y = torch.empty((b.m, k), dtype=torch.float32, device="cuda")
        for use_graph in (True, False, True):
            y.fill_(float("nan"))
            b.execute(x, y, use_graph=use_graph)
            b.check()
            assert (y.cpu().numpy() == want).all(), (launches, use_graph)
        b.close()


def test_batch_of_regular_members_is_one_launch(cuda_ok):
    """No run of long rows: no tile workers and no carry records."""
    import torch
    from benchmark_spmv_using_csr_gb300 import batch, gen
    a = gen.stencil3d(20, 21, 22, seed=3)
    a.val = gen.uniform_int(a.nnz, 8, 10) - 4.0
    b = batch.Batch([a, a], k=4)
    assert b.info()["launches"] == 1
    x = torch.ones((b.n, 4), dtype=torch.float32, device="cuda")
    y = torch.full((b.m, 4), float("nan"), dtype=torch.float32, device="cuda")
    b.execute(x, y)
    b.check()
    row = np.repeat(np.arange(a.m), np.diff(a.row_ptr))
    want = np.bincount(row, a.val, a.m)
    assert (y.cpu().numpy() == np.tile(want, 2)[:, None]).all()
    b.close()
