"""The batched form over work lists: the kernel variant and the tiles of its tile workers, calls on changing
buffers, and the tuner on it."""
import numpy as np
import pytest

from benchmark_spmv_using_csr_gb300 import batch, gen

pytestmark = pytest.mark.gpu


def _us(b, x, y):
    """Microseconds per execute: the least of 5 runs of 20 after a first one."""
    import torch
    out = []
    for _ in range(6):
        e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        e0.record()
        for _ in range(20):
            b.execute(x, y)
        e1.record()
        torch.cuda.synchronize()
        out.append(e0.elapsed_time(e1) * 50)
    return min(out[1:])


@pytest.mark.parametrize("kind,k", [("wide", 1), ("wide", 2), ("long", 1)])
def test_long_rows_between_row_blocks_are_no_slower_than_the_one_kernel(cuda_ok, kind, k):
    """Long rows (512 near columns, or 300 to 1500 random ones) between 27-point stencils: over work
    lists the batch takes at most 1.1 times what the one tile kernel over all rows takes at 4 tiles
    per worker (a forced variant: the one that the rule chooses for the whole batch)."""
    import torch
    stencil = gen.stencil3d(60, 60, 60)
    rng = np.random.default_rng(3)
    other = (gen.blockdiag(12_288, 12_288, 512) if kind == "wide" else
             gen.from_row_lengths(rng.integers(300, 1500, 6000), 50_000, seed=9))
    b = batch.Batch([stencil, other] * 2, k=k)
    x = torch.rand(b.n, k, device="cuda")
    y = torch.empty(b.m, k, device="cuda")
    lists = _us(b, x, y)
    b.reschedule(16, 4, 4)
    info = b.info()
    b.set_variant(l2_only=info["x_l2_only"])  # the same variant, forced: the one tile kernel
    one = _us(b, x, y)
    b.check()
    b.close()
    assert lists <= 1.1 * one, (lists, one)


@pytest.mark.parametrize("rows,count,k", [(6000, 2, 1), (7000, 4, 1), (6000, 2, 8)])
def test_default_tiles_per_worker_of_long_rows(cuda_ok, rows, count, k):
    """Rows of 300 to 1500 random columns alone: the default schedule takes at most 1.05 times what 4
    tiles per worker take."""
    import torch
    rng = np.random.default_rng(3)
    a = gen.from_row_lengths(rng.integers(300, 1500, rows), 50_000, seed=9)
    b = batch.Batch([a] * count, k=k)
    x = torch.rand(b.n, k, device="cuda")
    y = torch.empty(b.m, k, device="cuda")
    default = _us(b, x, y)
    b.reschedule(16, 4, 4)
    four = _us(b, x, y)
    b.close()
    assert default <= 1.05 * four, (default, four)


@pytest.mark.parametrize("seg", [8, 16, 32])
@pytest.mark.parametrize("spread", [False, True])
@pytest.mark.parametrize("k", [1, 2, 4, 8])
def test_tile_workers_variants_bit_exact(cuda_ok, k, seg, spread):
    """Runs of long rows (the one-head chunk form at one right-hand side) with near and with random
    columns, beginning and ending inside a tile, with a few short and empty rows among them, between
    blocks of short even rows: against an exact sum."""
    import torch
    rng = np.random.default_rng(100 * k + seg + spread)

    def rows(lens, near):
        lens = np.asarray(lens)
        n = 3000
        a = gen.from_row_lengths(lens, n, seed=int(rng.integers(1 << 30)))
        if near:
            row = np.repeat(np.arange(a.m), np.diff(a.row_ptr))
            a.col = ((7 * row + np.arange(a.nnz) - a.row_ptr[row]) % n).astype(np.int32)
        a.val = rng.integers(-4, 5, a.nnz).astype(np.float64)
        return a

    lens = rng.integers(230, 1100, 301)
    lens[[0, 7, 150, 300]] = [0, 3, 1, 0]
    mats = [rows(np.full(3001, 27), True), rows(lens, not spread), rows(np.full(2000, 9), True),
            rows(lens[::-1], not spread), rows(np.full(6000, 32), True)]
    b = batch.Batch(mats, k=k, seg=seg)
    x_np = rng.integers(-4, 5, (b.n, k)).astype(np.float64)
    row = np.repeat(np.arange(b.m), np.diff(b.cat["row_ptr"]))
    want = np.stack([np.bincount(row, b.cat["val"] * x_np[b.cat["col"], i], b.m) for i in range(k)], 1)
    x = torch.from_numpy(x_np.astype(np.float32)).cuda()
    y = torch.empty((b.m, k), dtype=torch.float32, device="cuda")
    for use_graph in (True, False, True):
        y.fill_(float("nan"))
        b.execute(x, y, use_graph=use_graph)
        b.check()
        assert (y.cpu().numpy() == want).all(), use_graph
    b.close()


@pytest.mark.parametrize("k", [1, 8])
def test_changing_buffers_cost_no_capture_per_call(cuda_ok, k):
    """Two x / y pairs in turn with use_graph: exact on both, and a call takes at most 1.25 times what
    a direct launch takes, and 3 us (a capture and instantiation per call would be 15 us and more);
    the same pair over and over is a graph replay, exact too, also after the other pair."""
    import torch
    rng = np.random.default_rng(k)
    mats = [gen.stencil2d(80, 80), gen.powerlaw(5000, seed=2), gen.blockdiag(4096, 4096, 32)]
    for a in mats:
        a.val = rng.integers(-4, 5, a.nnz).astype(np.float64)
    b = batch.Batch(mats, k=k)
    row = np.repeat(np.arange(b.m), np.diff(b.cat["row_ptr"]))
    pairs = []
    for _ in range(2):
        x = rng.integers(-4, 5, (b.n, k)).astype(np.float64)
        want = np.stack([np.bincount(row, b.cat["val"] * x[b.cat["col"], i], b.m) for i in range(k)], 1)
        pairs.append((torch.from_numpy(x.astype(np.float32)).cuda(),
                      torch.empty((b.m, k), dtype=torch.float32, device="cuda"), want))

    def per_call(use_graph, turn):
        out = []
        for _ in range(6):
            torch.cuda.synchronize()
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            for i in range(40):
                x, y, _ = pairs[i % 2 if turn else 0]
                b.execute(x, y, use_graph=use_graph)
            e1.record()
            torch.cuda.synchronize()
            out.append(e0.elapsed_time(e1) * 25)
        return min(out[1:])

    direct = per_call(False, True)
    turns = per_call(True, True)
    per_call(True, False)
    for i in (0, 1, 1, 1, 0, 0, 1, 0):
        x, y, want = pairs[i]
        y.fill_(float("nan"))
        b.execute(x, y)
        b.check()
        assert (y.cpu().numpy() == want).all(), i
    b.close()
    assert turns <= 1.25 * direct + 3.0, (turns, direct)


@pytest.mark.parametrize("k", [1, 8])
def test_autotune_times_one_schedule_once(cuda_ok, k):
    """Candidates that differ only in what work lists do not use have one time: the warps per CTA
    where tile workers run beside row blocks, everything where there are none; the pick is the first
    of the fastest."""
    import torch
    stencil = gen.stencil3d(20, 21, 22)
    for mats, tiles in (([stencil, gen.powerlaw(20_000, seed=3)] * 2, True), ([stencil] * 2, False)):
        b = batch.Batch(mats, k=k)
        x = torch.rand(b.n, k, device="cuda")
        y = torch.empty(b.m, k, device="cuda")
        ms, best = batch.autotune(b, x, y, warmup=1, reps=3)
        cands = batch.tune_candidates()
        for i, (seg, tpw, warps) in enumerate(cands):
            assert ms[i] == ms[cands.index((seg, tpw, 4))]
            assert tiles or ms[i] == ms[0]
        assert best == int(np.argmin(ms))
        b.close()
